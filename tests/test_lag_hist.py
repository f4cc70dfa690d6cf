"""CPU checks of the resident-history lag kernel's launch tables and barrier protocol
(cuda_multiddm_b200/csrc/lag_hist.cuh, lag_hist_host.hpp, built through
tests/hist_table_probe.cu): for the windows of both estimators and for random windows with
holes, every existing pair is formed exactly once and by the same kind of sum as the ring
kernel's table asks for, the copies fill exactly the rows that hold a frame, and a replay of
the barriers under random interleavings never reads a row that holds another block's data.
"""
from __future__ import annotations

import os
import random
import subprocess
from pathlib import Path

import pytest

from cuda_multiddm_b200.media import log_taus

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "cuda_multiddm_b200" / "csrc"
PROBE_SRC = ROOT / "tests" / "hist_table_probe.cu"
PROBE = ROOT / "tests" / "_build" / "hist_table_probe"
FUSE, MAX_SUB, STAGES, SLAB, X_ROWS = 4, 4, 11, 32, 32
LENGTH = (1, 1, FUSE)  # entries of a unit by kind
# elements per block, consumer warps, row buffers, register-frame buffers
SHAPES = ((32, 4, 3, 0), (32, 4, 1, 1), (16, 4, 1, 1), (16, 4, 2, 0), (16, 6, 1, 0), (16, 12, 1, 1))
SMEM_MAX = 232448
JS = (4, 8, 16, 20, 24, 30, 32)


@pytest.fixture(scope="module")
def probe() -> Path:
    deps = [PROBE_SRC] + [CSRC / f for f in ("lag_hist_host.hpp", "lag_hist.cuh", "lag_host.hpp", "lag.cuh")]
    if not PROBE.exists() or PROBE.stat().st_mtime < max(p.stat().st_mtime for p in deps):
        PROBE.parent.mkdir(parents=True, exist_ok=True)
        tmp = PROBE.with_name(f"{PROBE.name}.{os.getpid()}")
        subprocess.run(["nvcc", "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC),
                        str(PROBE_SRC), "-o", str(tmp)], check=True)
        os.replace(tmp, PROBE)
    return PROBE


def causal(shape, taus, n0, nreg, nsub, R):
    tmax, T, c = max(taus), len(taus), nreg * nsub
    slot = lambda f: f % R if f >= 0 else -1  # noqa: E731
    return dict(shape=shape, nreg=nreg, nsub=nsub, reg=[slot(n0 + j) for j in range(c)], ent_acc=list(range(T - 1, -1, -1)),
                ent_w=[tmax - taus[i] for i in range(T - 1, -1, -1)], pos=[slot(n0 - tmax + p) for p in range(c + tmax)])


def forward(shape, taus, nreg, nsub, R, rng):
    """The reference schedule's windows: the register frames open the position list."""
    labels = [rng.randrange(R) if rng.random() < 0.1 else p % R for p in range(nreg * nsub + max(taus))]
    return dict(shape=shape, nreg=nreg, nsub=nsub, reg=labels[:nreg * nsub], ent_acc=list(range(len(taus))), ent_w=list(taus),
                pos=labels)


def holes(shape, rng):
    """Random ascending windows over positions with missing frames and registers of their own."""
    nreg, T, R = rng.choice(JS + (1, 3, 17, 28)), rng.randint(1, 40), 900
    w = sorted(rng.sample(range(0, 400), T))
    pos = [-1 if rng.random() < 0.05 else rng.randrange(R) for _ in range(400 + nreg)]
    reg = [-1 if rng.random() < 0.1 else rng.randrange(R) for _ in range(nreg)]
    return dict(shape=shape, nreg=nreg, nsub=1, reg=reg, ent_acc=list(range(T)), ent_w=w, pos=pos)


def cases():
    rng = random.Random(11)
    out = []
    for shape in SHAPES:
        for taus in ([1], list(range(1, 21)), log_taus(1, 100, 48), log_taus(1, 500, 64), [3, 5, 6, 7, 8, 9, 40, 41, 44]):
            for nreg, nsub in ((32, 1), (32, 2), (30, 1), (30, 2), (28, 1), (16, 4), (8, 3), (17, 1), (4, 1), (1, 1)):
                for n0 in (0, 31, 77, 2000):
                    out.append(causal(shape, taus, n0, nreg, nsub, max(taus) + 91))
                out.append(forward(shape, taus, nreg, nsub, max(taus) + 64, rng))
        out += [holes(shape, rng) for _ in range(40)]
    return out


def tables(probe, cs):
    text = "".join(" ".join(map(str, [*c["shape"], c["nreg"], c["nsub"], len(c["ent_acc"]), len(c["pos"])] + c["reg"] +
                                c["ent_acc"] + c["ent_w"] + c["pos"])) + "\n" for c in cs)
    lines = subprocess.run([str(probe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(lines) == len(cs)
    out = [(c, [int(v) for v in ln.split()]) for c, ln in zip(cs, lines) if not ln.startswith("ERR")]
    for c, ln in zip(cs, lines):  # refused only where the rows cannot fit, or registers are not among them
        if ln.startswith("ERR"):
            assert "fit" in ln and (len(c["pos"]) + 64) * c["shape"][0] * 8 > SMEM_MAX * 0.9, ln
    return out


def parse(c, line):
    t = line[2:]
    EB, CW, *_ = c["shape"]
    halves = 32 // EB
    nreg, nsub, nrows, npiece, nx, reg_row, variants, buffers, steps_at, ints, x_bytes, arrive = t[:12]
    assert ints == len(t) and (nreg, nsub) == (c["nreg"], c["nsub"]) and 1 <= buffers <= 4
    assert EB * 8 * (buffers * nrows + (2 * X_ROWS if nx else 0)) < line[0] <= SMEM_MAX
    sub_stages, stage_bytes = t[12:12 + MAX_SUB], t[12 + MAX_SUB:12 + MAX_SUB + STAGES]
    p = 12 + MAX_SUB + STAGES
    assert arrive == 1 and sub_stages[:nsub] == sorted(sub_stages[:nsub]) and sub_stages[nsub - 1] <= STAGES
    raw, p = [t[p + 2 * i:p + 2 * i + 2] for i in range(npiece + nx)], p + 2 * (npiece + nx)
    lptr = t[p:p + variants * CW + 1]
    assert p + variants * CW + 1 <= steps_at and steps_at % 4 == 0
    steps = [t[i:i + 4] for i in range(steps_at, ints, 4)]
    assert len(steps) == lptr[-1] * halves and lptr == sorted(lptr)
    pieces = [(a & 0xFFFFF, ((a >> 20) & 31) + 1, b & 0xFFFF, b >> 16) for a, b in raw]
    rows, xrows = [None] * nrows, [None] * X_ROWS
    for i, (slot, n, row, stage) in enumerate(pieces):
        assert slot // SLAB == (slot + n - 1) // SLAB and 0 <= stage < STAGES
        into = rows if i < npiece else xrows
        for k in range(n):
            assert into[row + k] is None
            into[row + k] = slot + k
    pieces = pieces[:npiece]
    assert pieces == sorted(pieces, key=lambda q: q[2]) and [q[3] for q in pieces] == sorted(q[3] for q in pieces)
    assert stage_bytes == [128 * sum(q[1] for q in pieces if q[3] == s) for s in range(STAGES)]
    assert x_bytes == 128 * sum(r is not None for r in xrows) and all(q[3] < sub_stages[nsub - 1] for q in pieces)
    return dict(nrows=nrows, npiece=npiece, nx=nx, reg_row=reg_row, variants=variants, buffers=buffers, lptr=lptr,
                steps=steps, rows=rows, xrows=xrows, halves=halves, warps=CW, pieces=pieces, sub_stages=sub_stages)


def rows_of(t, stages):
    """The rows the first `stages` stages bring."""
    return {r + k for _, n, r, st in t["pieces"] if st < stages for k in range(n)}


def expected_runs(c, b):
    """First entries of the fused runs, by the ring kernel's rule."""
    nreg, w = c["nreg"], c["ent_w"]
    full = [nreg in JS and all(c["reg"][b * nreg + j] >= 0 and c["pos"][w[i] + b * nreg + j] >= 0 for j in range(nreg))
            for i in range(len(w))]
    out, i = set(), 0
    while i < len(w):
        if i + FUSE <= len(w) and all(full[i + r] and w[i + r] == w[i] + r for r in range(FUSE)):
            out.add(i)
            i += FUSE
        else:
            i += 1
    return out


def steps_of(t, warps, b):
    """The steps (a unit per half) of the given warps in sub-batch b."""
    for w in warps:
        v = (b if t["variants"] > 1 else 0) * t["warps"] + w
        for s in range(t["lptr"][v], t["lptr"][v + 1]):
            yield [(row // 128, acc // 128, mask // 128 if info & 3 == 2 else mask, info)
                   for row, acc, mask, info in t["steps"][s * t["halves"]:(s + 1) * t["halves"]]]


def check_pairs(c, t):
    nreg, entry = c["nreg"], {a: i for i, a in enumerate(c["ent_acc"])}
    for b in range(c["nsub"]):
        for j in range(nreg):  # register frames: their buffer, or resident rows that have landed
            want = c["reg"][b * nreg + j]
            if b == 0 and t["nx"]:
                assert want < 0 or t["xrows"][j] == want
            else:
                r = t["reg_row"] + b * nreg + j
                assert want < 0 or (t["rows"][r] == want and r in rows_of(t, t["sub_stages"][b]))
        seen, runs = {}, set()
        for step in steps_of(t, range(t["warps"]), b):
            assert len({info & 3 for *_, info in step}) == 1
            for row, acc, mask, info in step:
                kind, row = info & 3, row + b * nreg
                ready = rows_of(t, max((info >> 4) & 15, t["sub_stages"][b] if b and t["variants"] == 1 or not t["nx"]
                                       else 0))
                assert kind or mask
                if not kind:
                    assert {row + j for j in range(nreg) if (mask >> j) & 1} <= ready
                if kind:  # every row read has landed
                    assert set(range(row, row + nreg + (LENGTH[kind] - 1))) <= ready
                if kind == 1:
                    assert mask & 0xFFFFFFFF == (1 << nreg) - 1
                if not info & 4:
                    continue
                for r in range(LENGTH[kind]):
                    i = entry[acc + r * mask] if kind >= 2 else entry[acc]
                    if kind >= 2 and r % FUSE == 0:
                        runs.add(i)
                    for j in range(nreg):
                        if kind == 0 and not (mask >> j) & 1:
                            continue
                        want = c["pos"][c["ent_w"][i] + b * nreg + j]
                        assert want >= 0 and row + r + j in ready and t["rows"][row + r + j] == want
                        assert (i, j) not in seen
                        seen[(i, j)] = True
        assert runs == expected_runs(c, b)
        pairs = {(i, j) for i in range(len(c["ent_acc"])) for j in range(nreg)
                 if c["reg"][b * nreg + j] >= 0 and c["pos"][c["ent_w"][i] + b * nreg + j] >= 0}
        assert set(seen) == pairs


def test_tables_form_every_pair_once(probe):
    cs = cases()
    for c, line in tables(probe, cs):
        check_pairs(c, parse(c, line))


class Bar:
    """An mbarrier: phase parity flips when `count` arrivals (and no pending bytes) are in."""

    def __init__(self, count):
        self.count, self.left, self.pending, self.phase = count, count, 0, 0

    def arrive(self, pending=0):
        assert self.left > 0
        self.left -= 1
        self.pending += pending
        self.settle()

    def land(self, n):
        self.pending -= n
        self.settle()

    def settle(self):
        if self.left == 0 and self.pending == 0:
            self.left, self.phase = self.count, self.phase + 1

    def done(self, parity):
        return (self.phase & 1) != parity


def replay(c, t, blocks, rng):
    nsub, nbuf, warps, nst = c["nsub"], t["buffers"], t["warps"], t["sub_stages"][c["nsub"] - 1]
    full = [[Bar(1) for _ in range(nst)] for _ in range(nbuf)]
    empty = [[Bar(warps) for _ in range(nst)] for _ in range(nbuf)]
    xfull, xempty, sub_done = [Bar(1), Bar(1)], [Bar(warps), Bar(warps)], Bar(warps)
    held = [[None] * nst for _ in range(nbuf)]  # the block whose rows a stage of a buffer holds
    xheld = [None, None]
    stage_of = {r + k: st for _, n, r, st in t["pieces"] for k in range(n)}
    flying = []

    def producer():
        def issue_x(n):
            if t["nx"] and n < blocks:
                while n > 1 and not xempty[n & 1].done(((n >> 1) - 1) & 1):
                    yield
                xheld[n & 1] = None
                xfull[n & 1].arrive(1)
                flying.append((xheld, n & 1, n, xfull[n & 1]))

        yield from issue_x(0)
        for n in range(blocks):
            yield from issue_x(n + 1)
            buf, use = n % nbuf, n // nbuf
            for st in range(nst):
                while use > 0 and not empty[buf][st].done((use - 1) & 1):
                    yield
                held[buf][st] = None
                full[buf][st].arrive(1)
                flying.append((held[buf], st, n, full[buf][st]))
                yield

    def consumer(warp):
        for n in range(blocks):
            buf, have, released, parity = n % nbuf, 0, 0, (n // nbuf) & 1

            def stages(need):
                nonlocal have
                while have < need:
                    while not full[buf][have].done(parity):
                        yield
                    have += 1

            while t["nx"] and not xfull[n & 1].done((n >> 1) & 1):
                yield
            for b in range(nsub):
                if b or not t["nx"]:
                    yield from stages(t["sub_stages"][b])
                if b == 0 and t["nx"]:
                    assert xheld[n & 1] == n
                    xempty[n & 1].arrive()
                else:
                    for j in range(c["nreg"]):
                        if c["reg"][b * c["nreg"] + j] >= 0:
                            assert held[buf][stage_of[t["reg_row"] + b * c["nreg"] + j]] == n
                for step in steps_of(t, [warp], b):
                    yield from stages(step[0][3] >> 4 & 15)
                    if b == nsub - 1:
                        for st in range(released, step[0][3] >> 8):
                            empty[buf][st].arrive()
                        released = max(released, step[0][3] >> 8)
                    for row, _, mask, info in step:
                        row += b * c["nreg"]
                        rows = (range(row, row + c["nreg"] + (LENGTH[info & 3] - 1)) if info & 3 else
                                [row + j for j in range(c["nreg"]) if (mask >> j) & 1])
                        assert all(held[buf][stage_of[r]] == n for r in rows)
                    yield
                if t["variants"] > 1 and b < nsub - 1:
                    sub_done.arrive()
                    while not sub_done.done((n * (nsub - 1) + b) & 1):
                        yield
            yield from stages(nst)
            for st in range(released, nst):
                empty[buf][st].arrive()
            yield

    actors = [producer()] + [consumer(w) for w in range(warps)]
    idle = 0
    while actors:
        if flying and rng.random() < 0.4:
            hold, i, n, bar = flying.pop(rng.randrange(len(flying)))
            hold[i] = n
            bar.land(1)
            idle = 0
        a = rng.choice(actors)
        try:
            next(a)
        except StopIteration:
            actors.remove(a)
            idle = 0
        idle += 1
        assert idle < 200000, "the protocol does not advance"


def test_barrier_protocol_replay(probe):
    rng = random.Random(5)
    cs = [c for c in cases() if rng.random() < 0.02]
    for c, line in tables(probe, cs):
        t = parse(c, line)
        if t["npiece"]:
            replay(c, t, 4, rng)


@pytest.mark.gpu
@pytest.mark.parametrize("side,scales,taus,chunk,calls", [
    (64, [64, 32], log_taus(1, 40, 12), 7, (1, 6, 33, 20)),          # odd pieces, first frames without partners
    (256, [256, 16], log_taus(1, 260, 64), 32, (40, 300, 5)),        # 16-element blocks, two buffers
    (512, [512, 256, 128, 64], log_taus(1, 90, 40), 30, (200, 64, 31)),  # two batches per launch
    (512, [512, 256, 128], log_taus(1, 620, 64), 17, (680, 130)),    # two CTAs per SM, two batches
])
def test_sums_match_float64(side, scales, taus, chunk, calls):
    """Every lag sum of every spectrum element against the same sum in float64 over the engine's own
    spectra: the launches' FP32 sums of up to 32 pairs round at most 2 * 32 times each (a difference,
    a square and a sum per component), the Kahan sums over launches twice; so 1e-5 of the sum of the
    exact squares bounds the error with an order of magnitude to spare."""
    import numpy as np
    import torch
    from cuda_multiddm_b200 import Engine, EngineConfig
    rng = np.random.default_rng(side + chunk)
    n = sum(calls)
    frames = rng.integers(0, 256, (n, side, side), dtype=np.uint8)
    with Engine(EngineConfig(frame_width=side, frame_height=side, scales=scales, taus=taus, lambdas=[4.0, 8.0],
                             chunk_frames=chunk)) as eng:
        spec, done = [], 0
        for c in calls:
            eng.submit(frames[done:done + c])
            done += c
        got = eng.accumulators()
    x = torch.from_numpy(frames.astype(np.float64)).cuda()
    F = torch.cat([torch.fft.rfft2(x.view(n, side // s, s, side // s, s).permute(0, 1, 3, 2, 4)).reshape(n, -1)
                   for s in sorted(scales, reverse=True)], 1)
    for i, tau in enumerate(taus):
        want = torch.zeros(F.shape[1], dtype=torch.float64, device="cuda")
        for t in range(tau, n):
            want += torch.view_as_real(F[t] - F[t - tau]).square().sum(-1)
        err = (torch.from_numpy(got[i]).cuda() - want).abs()
        scale = want + (n - tau) * (1e-6 * F.abs().amax()) ** 2 + 1e-30  # spectra: 1e-6 of the largest value
        spectra = 2 * torch.sqrt(want * max(n - tau, 0)) * 2e-6 * F.abs().amax()  # their effect on a sum
        assert bool((err <= 1e-5 * scale + spectra).all()), (tau, float((err / scale).max()))
