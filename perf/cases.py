"""What users of this framework have it do, as measurable cases.

Every case is one pass through the public entry points: frames in, the image structure
function (ISF) out. Its sizes come from the repository's configurations (bench.py's c1..c4, the
serving mix, the tests) and their neighbourhood:

  kind "stream"  one Engine that stays open, as a camera program or an analysis of recorded
                 frames keeps it. `history` frames are in the ring already (their sums reset),
                 one pass submits `frames` more, `submit` at a time, and takes the result: once
                 at the end (result "end"), after every submit through finalize_async with
                 three results in flight ("live"), or with the decay fits ("fit").
  kind "compat"  run_ddm on a video in host memory with the reference's own schedule: engine
                 opened, video analysed, engine closed, as one call.
  kind "static"  the lag accumulation on the caller's own ring and accumulators.
  kind "server"  one chunk of every stream of a Server, from submit to poll.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cuda_multiddm_b200 import Engine, EngineConfig, Server, lib, log_lambdas, log_taus, run_ddm

TOLERANCE = 1.2


def _stream(name, side, scales, taus, lambdas, **kw):
    """A stream case: taus (first, last, count) and lambdas (first, last, count) are log-spaced."""
    case = dict(name=name, kind="stream", width=side, height=side, x=0, y=0, pixel="u8",
                scales=",".join(map(str, scales)), tau_lo=taus[0], tau_hi=taus[1], tau_n=taus[2],
                lambda_lo=float(lambdas[0]), lambda_hi=float(lambdas[1]), lambda_n=lambdas[2], chunk=30,
                history=0, frames=30, submit=30, device=True, result="end")
    case.update(kw)
    return case


def listed():
    c2 = (1024, (1024, 512, 256, 128), (1, 500, 64), (2, 512, 30))
    return [
        # The smallest call in use: a 256^2 camera stream, the updated ISF after every 30-frame
        # chunk from pinned host memory. Launches and host work count.
        _stream("live_256", 256, (256,), (1, 20, 20), (4, 128, 10), history=60, device=False),
        # A short recorded 256^2 video in one call (configuration c1).
        _stream("video_256", 256, (256,), (1, 20, 20), (4, 128, 10), frames=200, submit=200),
        # The headline configuration as a camera program runs it: chunks of 30 frames from pinned
        # host memory, a live result for each (the end-to-end leg of the benchmark).
        _stream("live_1024", *c2, history=510, frames=120, device=False, result="live"),
        # The headline configuration as the benchmark's device-resident leg runs it: frames in GPU
        # memory, 30 per call, one result.
        _stream("chunks_1024", *c2, history=510, frames=240),
        # The same video of 480 frames handed over in one call, on a new engine the first time.
        _stream("video_1024", *c2, frames=480, submit=480),
        # Many small tiles (configuration c3 with a shorter longest lag): 5461 tiles a frame.
        _stream("fine_2048", 2048, (2048, 1024, 512, 256, 128, 64, 32), (1, 100, 48), (2, 1024, 40), history=120,
                frames=60),
        # 12-bit camera data in 16-bit pixels (configuration c4 with a shorter longest lag).
        _stream("highbit_2048", 2048, (2048, 1024, 512, 256), (1, 200, 64), (2, 1024, 30), history=210, frames=60,
                pixel="u16"),
        # A region of interest at an odd offset of a larger camera frame, odd chunk and list sizes.
        _stream("roi_512", 512, (512, 128, 32), (1, 90, 37), (3, 200, 13), width=1280, height=960, x=37, y=11,
                chunk=17, submit=17, frames=17, history=102, device=False),
        # A live result with its decay rates and diffusion coefficients (the CLI's -D).
        _stream("fit_512", 512, (512, 256, 128, 64), (1, 100, 64), (2, 128, 30), history=120, device=False,
                result="fit"),
        # run_ddm with its defaults: the reference's schedule on a video in host memory.
        dict(name="compat_512", kind="compat", side=512, scales="512,256,128", tau_lo=1, tau_hi=100, tau_n=40,
             lambda_lo=2.0, lambda_hi=128.0, lambda_n=20, chunk=100, frames=300),
        # The allocation-free entry point on a caller's ring: 32 frames against 64 lags.
        dict(name="static_lag", kind="static", elements=531968, slots=600, frames=32, tau_lo=1, tau_hi=500, tau_n=64),
        # Serving: one chunk of each of 8 streams of mixed sizes through one server.
        dict(name="server_8", kind="server", streams=8, largest=1024, mix=5, chunk=30, history=90),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    pick = rng.random()
    if pick < 0.08:
        return dict(kind="static", elements=2 * logint(5000, 400000), slots=600, frames=rng.randint(1, 32), tau_lo=1,
                    tau_hi=logint(70, 500), tau_n=rng.randint(5, 64))
    if pick < 0.16:
        return dict(kind="server", streams=rng.randint(2, 8), largest=rng.choice((256, 512, 1024)),
                    mix=rng.randint(1, 10 ** 6), chunk=rng.choice((10, 25, 30, 32)), history=90)
    side = rng.choice((64, 128, 256, 512, 512, 1024, 1024, 2048))
    smaller = [s for s in (1024, 512, 256, 128, 64, 32, 16) if s < side]
    scales = [side] + [s for s in smaller if rng.random() < 0.5]
    if pick < 0.26:
        side = min(side, 512)
        scales = [side] + [s for s in scales if s < side]
        chunk = rng.randint(20, 120)
        tau_hi = rng.randint(10, chunk)
        return dict(kind="compat", side=side, scales=",".join(map(str, scales)), tau_lo=1, tau_hi=tau_hi,
                    tau_n=rng.randint(5, tau_hi), lambda_lo=2.0, lambda_hi=float(min(scales)),
                    lambda_n=rng.randint(3, 20), chunk=chunk, frames=chunk * rng.randint(2, 3))
    device = rng.random() < 0.5
    chunk = rng.choice((16, 20, 25, 30, 30, 32, 32, 48, 64))
    result = rng.choice(("end", "end", "end", "live", "fit"))
    calls = 1 if result == "fit" else rng.randint(1, 4)
    submit = chunk if result != "end" or rng.random() < 0.6 else logint(chunk, 300)
    elements = sum((side // s) ** 2 * s * (s // 2 + 1) for s in scales)
    tau_hi = logint(8, 700)
    while (tau_hi + 128) * elements * 8 > 16e9:  # three states fit the card
        tau_hi = tau_hi * 3 // 4
    tau_n = rng.randint(min(5, tau_hi), min(100, tau_hi))
    while calls * submit * elements * tau_n > 480 * 2112512 * 64:  # no more work than the largest listed case
        if submit > chunk:
            submit = max(chunk, submit // 2)
        elif calls > 1:
            calls -= 1
        else:
            tau_n = tau_n // 2
    x, y = (rng.randint(0, 40), rng.randint(0, 40)) if rng.random() < 0.3 else (0, 0)
    case = _stream("", side, scales, (1, tau_hi, tau_n), (2.0, float(side) / 2, rng.randint(3, 40)),
                   width=side + x + (rng.randint(0, 60) if x else 0), height=side + y, x=x, y=y, chunk=chunk,
                   history=rng.choice((0, min(tau_hi + 10, 510))), frames=calls * submit, submit=submit, device=device,
                   result=result, pixel=rng.choice(("u8", "u8", "u16")))
    del case["name"]
    return case


# ---- inputs ---------------------------------------------------------------------------------

def _video(gen, n, height, width, u16):
    """n frames [n, height, width] of Brownian Gaussian spots on a background with camera noise,
    as float32 on the GPU rounded to 8-bit (12-bit for u16) values."""
    spots = max(8, 4000 * height * width // (1024 * 1024))
    amplitude, background, top = (2000.0, 300.0, 4095.0) if u16 else (120.0, 20.0, 255.0)
    dev = torch.device("cuda")
    start = torch.rand((1, spots, 2), generator=gen, device=dev) * torch.tensor([height, width], device=dev)
    steps = torch.randn((n, spots, 2), generator=gen, device=dev)
    pos = (start + steps.cumsum(0)).round().long()
    cell = (pos[..., 0] % height) * width + pos[..., 1] % width
    taps = torch.exp(-0.5 * (torch.arange(-6, 7, device=dev) / 2.0) ** 2)
    out = torch.empty((n, height, width), dtype=torch.float32, device=dev)
    for f0 in range(0, n, 32):
        img = torch.zeros((min(32, n - f0), height * width), device=dev)
        img.scatter_add_(1, cell[f0:f0 + 32], torch.full_like(cell[f0:f0 + 32], amplitude, dtype=torch.float32))
        img = img.view(-1, height, width)
        for dim in (1, 2):
            img = sum(float(taps[6 + k]) * img.roll(k, dim) for k in range(-6, 7))
        img += background
        noise = torch.randn(img.shape, generator=gen, device=dev)
        img += noise * (img.sqrt() if u16 else 4.0)
        out[f0:f0 + 32] = img.round_().clamp_(0.0, top)
    return out


def _pixels(video, u16):
    """The frames as a camera delivers them: bytes [n, height, width * bytes per pixel]."""
    if u16:
        return video.to(torch.int16).view(torch.uint8)
    return video.to(torch.uint8)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (1 << 62))


def _lists(case):
    return ([int(s) for s in case["scales"].split(",")], log_taus(case["tau_lo"], case["tau_hi"], case["tau_n"]),
            log_lambdas(case["lambda_lo"], case["lambda_hi"], case["lambda_n"]))


def _stream_video(case, seed):
    return _video(_generator(seed), case["history"] + case["frames"], case["height"], case["width"],
                  case["pixel"] == "u16")


def _server_specs(case):
    """The streams of a server: side, scales, taus, lambdas as the serving benchmark draws them."""
    rng = np.random.default_rng(case["mix"])
    specs = []
    for _ in range(case["streams"]):
        side = int(rng.choice([s for s in (256, 512, 1024) if s <= case["largest"]]))
        scales = [side] + [s for s in (512, 256, 128, 64, 32) if s < side and rng.random() < 0.5]
        tau_max = int(rng.integers(30, 301))
        taus = log_taus(1, tau_max, int(rng.integers(20, min(100, tau_max) + 1)))
        specs.append((side, scales, taus, log_lambdas(2.0, float(min(scales)), int(rng.integers(5, 21)))))
    return specs


def _server_videos(case, seed):
    gen = _generator(seed)
    return [_video(gen, case["history"] + case["chunk"], side, side, False) for side, *_ in _server_specs(case)]


def _static_input(case, seed):
    gen = _generator(seed)
    ring = torch.randn((case["slots"], case["elements"], 2), generator=gen, device="cuda")
    ring *= 100.0 * torch.rand((1, case["elements"], 1), generator=gen, device="cuda") + 1.0
    taus = log_taus(case["tau_lo"], case["tau_hi"], case["tau_n"])
    first = case["tau_hi"] + 3
    a = [(first + j) % case["slots"] for j in range(case["frames"])]
    b = [[(first + j - t) % case["slots"] for j in range(case["frames"])] for t in taus]
    return ring, a, b


class _Open:
    """What a program keeps open; closed with the state."""

    def __init__(self, thing):
        self.thing = thing

    def __del__(self):
        self.thing.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "stream":
        u16 = case["pixel"] == "u16"
        raw = _pixels(_stream_video(case, seed), u16)
        scales, taus, lambdas = _lists(case)
        eng = Engine(EngineConfig(frame_width=case["width"], frame_height=case["height"], scales=scales, taus=taus,
                                  lambdas=lambdas, tolerance=TOLERANCE, chunk_frames=case["chunk"],
                                  bytes_per_pixel=2 if u16 else 1, pixel_mode="u16" if u16 else "byte0",
                                  x_offset=case["x"], y_offset=case["y"]))
        if case["history"]:
            torch.cuda.synchronize()
            eng.submit(raw[:case["history"]])
            eng.reset()
            eng.synchronize()
        frames = raw[case["history"]:]
        frames = frames.clone() if case["device"] else frames.cpu().pin_memory()
        state = {"case": case, "engine": eng, "keep": _Open(eng),
                 "calls": [frames[i:i + case["submit"]] for i in range(0, case["frames"], case["submit"])]}
        if case["result"] == "live":
            eng.set_async_depth(4)
            state["results"] = [eng.pinned_isf_buffer() for _ in state["calls"]]
        torch.cuda.synchronize()
        return state
    if kind == "compat":
        video = _video(_generator(seed), case["frames"], case["side"], case["side"], False)
        return {"case": case, "video": _pixels(video, False).cpu().numpy(), "lists": _lists(case)}
    if kind == "static":
        ring, a, b = _static_input(case, seed)
        acc = torch.zeros((len(b), case["elements"], 2), device="cuda")
        torch.cuda.synchronize()
        return {"case": case, "ring": ring, "acc": acc, "a": np.asarray(a, np.int32), "b": np.asarray(b, np.int32)}
    specs = _server_specs(case)
    server = Server(hbm_budget_bytes=24 << 30, max_streams=case["streams"])
    keep = _Open(server)
    ids = [server.add_stream(EngineConfig(frame_width=side, frame_height=side, scales=scales, taus=taus,
                                          lambdas=lambdas, tolerance=TOLERANCE, chunk_frames=case["chunk"]))
           for side, scales, taus, lambdas in specs]
    videos = [_pixels(v, False).cpu().pin_memory() for v in _server_videos(case, seed)]
    for f0 in range(0, case["history"], case["chunk"]):
        for sid, v in zip(ids, videos):
            n = min(case["chunk"], case["history"] - f0)
            server.submit_pinned(sid, v[f0:].data_ptr(), n)
        server.step()
        server.wait()
        for sid in ids:
            server.poll(sid)
    return {"case": case, "server": server, "keep": keep, "ids": ids, "videos": videos,
            "chunks": [v[case["history"]:] for v in videos]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "stream":
        eng = state["engine"]
        if case["result"] == "live":
            for frames, isf in zip(state["calls"], state["results"]):
                eng.submit(frames)
                eng.finalize_async(isf)
            eng.wait_isf()
            return state["results"]
        for frames in state["calls"]:
            eng.submit(frames)
        eng.finalize()
        isf = eng.isf()
        return {"isf": isf, "fit": eng.fit()} if case["result"] == "fit" else isf
    if kind == "compat":
        scales, taus, lambdas = state["lists"]
        isf, _ = run_ddm(state["video"], scales, taus, lambdas, tolerance=TOLERANCE, chunk_frames=case["chunk"])
        return {str(s): v for s, v in isf.items()}
    if kind == "static":
        ring, acc, a, b = state["ring"], state["acc"], state["a"], state["b"]
        status = lib().ddm_lag_accumulate_static(ring.data_ptr(), ring.shape[0], ring.shape[1], acc.data_ptr(),
                                                 a.ctypes.data, a.size, b.ctypes.data, b.shape[0],
                                                 torch.cuda.current_stream().cuda_stream)
        if status:
            raise RuntimeError(lib().ddm_last_error().decode())
        return acc
    server = state["server"]
    for sid, frames in zip(state["ids"], state["chunks"]):
        server.submit_pinned(sid, frames.data_ptr(), frames.shape[0])
    server.step()
    server.wait()
    return [server.poll(sid)[1] for sid in state["ids"]]


# ---- work -----------------------------------------------------------------------------------

def _stream_work(side, scales, taus, lambda_n, bpp, history, frames, results, live_state):
    """Bytes and operations of analysing `frames` frames after `history` others: the pixels read
    and each result written once; where a stream stays open its state counts too: the new
    spectra are written, each older spectrum that a lag reaches is read and the sums are read
    and written, once. Operations: 2.5 N log2 N per real 2-D transform of N values, and 6 per
    pair and spectrum value (two subtractions, two products, two sums)."""
    elements = sum((side // s) ** 2 * s * (s // 2 + 1) for s in scales)
    older = len({t - tau for tau in taus for t in range(history, history + frames) if 0 <= t - tau < history})
    pairs = sum(max(0, min(frames, history + frames - tau)) for tau in taus)
    tiles = sum((side // s) ** 2 for s in scales)
    size = side * side * frames * bpp + 8 * tiles * lambda_n * len(taus) * results
    if live_state:
        size += 8 * elements * (frames + older + 2 * len(taus))
    transforms = sum(2.5 * side * side * math.log2(s * s) for s in scales) * frames
    return {"bytes": float(size), "flops": transforms + 6.0 * elements * pairs}


def work(case):
    kind = case["kind"]
    if kind == "static":
        taus = log_taus(case["tau_lo"], case["tau_hi"], case["tau_n"])
        older = len({j - t for t in taus for j in range(case["frames"])} | set(range(case["frames"])))
        return {"bytes": 8.0 * case["elements"] * (older + 2 * len(taus)),
                "flops": 6.0 * case["elements"] * case["frames"] * len(taus)}
    if kind == "server":
        parts = [_stream_work(side, scales, taus, len(lambdas), 1, case["history"], case["chunk"], 1, True)
                 for side, scales, taus, lambdas in _server_specs(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    scales, taus, _ = _lists(case)
    if kind == "compat":
        w = _stream_work(case["side"], scales, taus, case["lambda_n"], 1, 0, case["frames"], 1, False)
        return w
    results = len(range(0, case["frames"], case["submit"])) if case["result"] == "live" else 1
    return _stream_work(max(scales), scales, taus, case["lambda_n"], 2 if case["pixel"] == "u16" else 1,
                        case["history"], case["frames"], results, True)


# ---- the same in 64 bits -----------------------------------------------------------------------

def _annuli(s, lambdas):
    """[s * (s/2 + 1), lambda] of 0 and 1: the wave vectors with q <= |k| <= q * tolerance, q =
    s / lambda, decided in the reference's single precision."""
    y = np.arange(s)
    ys = (y + s // 2) % s - s // 2
    x = np.arange(s // 2 + 1)
    xs = (x + s // 2) % s - s // 2
    r2 = (xs[None, :] ** 2 + ys[:, None] ** 2).astype(np.float32).reshape(-1)
    tol2 = np.float32(TOLERANCE) * np.float32(TOLERANCE)
    cols = []
    for lam in lambdas:
        q = np.float32(s) / np.float32(lam)
        ratio = r2 / np.float32(q * q)
        cols.append((ratio >= np.float32(1.0)) & (ratio <= tol2))
    return torch.from_numpy(np.stack(cols, 1)).cuda()


def _exact_isf(video, scales, taus, lambdas, marks, pairs_of, norm_of):
    """The ISF at each mark (a number of frames) in double precision, flat as the engine returns
    it. pairs_of(tau, lo, hi): the (later, earlier) frame indices that frames lo .. hi-1 add."""
    n, side = video.shape[0], video.shape[1]
    out = [[] for _ in marks]
    for s in sorted(scales, reverse=True):
        side_n, width = side // s, s // 2 + 1
        tiles = side_n * side_n
        spec = torch.empty((n, tiles, s * width), dtype=torch.complex128, device="cuda")
        for f in range(n):
            t = video[f].double().view(side_n, s, side_n, s).permute(0, 2, 1, 3)
            spec[f] = torch.fft.rfft2(t).reshape(tiles, s * width)
        mask = _annuli(s, lambdas).double()
        count = mask.sum(0)
        isf = torch.zeros((len(marks), tiles, len(lambdas), len(taus)), dtype=torch.float64, device="cuda")
        for i, tau in enumerate(taus):
            total = torch.zeros((tiles, s * width), dtype=torch.float64, device="cuda")
            lo = 0
            for m, hi in enumerate(marks):
                for a, b in pairs_of(tau, lo, hi):
                    d = torch.view_as_real(spec[a] - spec[b])
                    total += d.square_().sum(-1)
                lo = hi
                value = 2.0 * (total @ mask) / float(s) ** 4 / count
                norm = norm_of(tau, hi)
                isf[m, :, :, i] = torch.where(count > 0, value / norm if norm else 0.0 * value, torch.zeros(()).double().cuda())
        for m in range(len(marks)):
            out[m].append(isf[m].reshape(-1).cpu().numpy())
        del spec
    return [np.concatenate(o) for o in out]


def _exact_stream(video, scales, taus, lambdas, first, marks):
    """Every pair whose later frame is one of first .. mark-1, each lag over its number of pairs."""
    return _exact_isf(video, scales, taus, lambdas, marks,
                      lambda tau, lo, hi: [(t, t - tau) for t in range(max(lo, first, tau), hi)],
                      lambda tau, hi: max(0, hi - max(first, tau)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "static":
        ring, a, b = _static_input(case, seed)
        out = torch.zeros((len(b), case["elements"], 2), dtype=torch.float64, device="cuda")
        regs = ring[torch.tensor(a, device="cuda")].double()
        for t, row in enumerate(b):  # {sum, compensation}: the limit of the compensation is 0
            d = ring[torch.tensor(row, device="cuda")].double() - regs
            out[t, :, 0] = d.square_().sum((0, 2))
        return out
    if kind == "server":
        return [_exact_stream(v, scales, taus, lambdas, 0, [v.shape[0]])[0]
                for v, (_, scales, taus, lambdas) in zip(_server_videos(case, seed), _server_specs(case))]
    scales, taus, lambdas = _lists(case)
    if kind == "compat":
        # The reference's pairing for a whole number (>= 2) of chunks: frame t with t + tau; past
        # the end of the video its buffers still hold the frames of two chunks before.
        n, chunk, side = case["frames"], case["chunk"], case["side"]
        video = _video(_generator(seed), n, side, side, False)
        flat, = _exact_isf(video, scales, taus, lambdas, [n],
                           lambda tau, lo, hi: [(t, t + tau if t + tau < n else t + tau - 2 * chunk)
                                                for t in range(lo, hi)], lambda tau, hi: n)
        out, off = {}, 0
        for s in sorted(scales, reverse=True):
            shape = ((side // s) ** 2, len(lambdas), len(taus))
            size = int(np.prod(shape))
            out[str(s)] = flat[off:off + size].reshape(shape)
            off += size
        return out
    if case["frames"] * max(scales) ** 2 * len(scales) * len(taus) > 480 * 1024 ** 2 * 4 * 64 * 2:
        return None
    side = max(scales)
    video = _stream_video(case, seed)[:, case["y"]:case["y"] + side, case["x"]:case["x"] + side].contiguous()
    first = case["history"]
    marks = [first + case["frames"]]
    if case["result"] == "live":
        marks = [first + min(i + case["submit"], case["frames"]) for i in range(0, case["frames"], case["submit"])]
    isf = _exact_stream(video, scales, taus, lambdas, first, marks)
    if case["result"] == "live":
        return isf
    if case["result"] == "fit":
        return {"isf": isf[0], "fit": None}
    return isf[0]
