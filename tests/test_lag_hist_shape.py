"""An engine that takes the resident-history lag kernel stays on it, so no launch of it may outgrow the
shape chosen for its full launches (CPU, through tests/hist_shape_probe.cu): partial launches form no fused
runs, the first launches of a stream miss partners, pairs of batches carry two lists."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

import pytest

from cuda_multiddm_b200.media import log_taus

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "cuda_multiddm_b200" / "csrc"
SRC = ROOT / "tests" / "hist_shape_probe.cu"
PROBE = ROOT / "tests" / "_build" / "hist_shape_probe"


@pytest.fixture(scope="module")
def probe() -> Path:
    deps = [SRC] + [CSRC / f for f in ("lag_hist_host.hpp", "lag_hist.cuh", "lag_host.hpp", "lag.cuh", "layout.cuh")]
    if not PROBE.exists() or PROBE.stat().st_mtime < max(p.stat().st_mtime for p in deps):
        PROBE.parent.mkdir(parents=True, exist_ok=True)
        tmp = PROBE.with_name(f"{PROBE.name}.{os.getpid()}")
        subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC),
                        str(SRC), "-o", str(tmp)], check=True)
        os.replace(tmp, PROBE)
    return PROBE


def run(probe, engines):
    """[(elements per block, launches, refused) per batch count] of each (compat, batch, R, n0 step, count step, taus)."""
    text = "".join(" ".join(map(str, [int(c), b, R, ns, cs, len(taus), *taus])) + "\n" for c, b, R, ns, cs, taus in engines)
    lines = subprocess.run([str(probe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(lines) == len(engines)
    out = []
    for ln in lines:
        v = [int(x) for x in ln.split()]
        out.append([tuple(v[i:i + 3]) for i in range(0, len(v), 3)])
    return out


def lists():
    """Lists whose rows come near what a CTA can hold, and ordinary ones."""
    out = [list(range(1, n + 1)) for n in (20, 300, 1400, 1500, 1560, 1582, 1600, 1640, 1700, 1723, 1760)]
    out += [list(range(1, n, 2)) for n in (1552, 1600, 1643)] + [list(range(1, n, 5)) for n in (1665, 1704)]
    out += [list(range(1, n, 8)) for n in (1696, 1751)] + [log_taus(1, n, 200) for n in (1600, 1717, 1731, 1760)]
    return out + [log_taus(1, 500, 64), log_taus(1, 100, 48), log_taus(1, 1730, 64), [1, 2, 3, 5, 8, 13, 40, 90, 200]]


@pytest.mark.parametrize("batch", [32, 30])
def test_no_launch_of_a_chosen_shape_is_refused(probe, batch):
    engines = [(False, batch, taus[-1] + 2 * batch, 131, 10, taus) for taus in lists()]
    for (_, _, _, _, _, taus), shapes in zip(engines, run(probe, engines)):
        for eb, tried, refused in shapes:
            assert refused == 0 and (eb == 0 or tried > 0), (taus[-1], len(taus), shapes)


def test_no_launch_of_the_reference_schedule_is_refused(probe):
    engines = [(True, 32, 2 * taus[-1] + 100, 307, 10, taus) for taus in lists()]
    for (_, _, _, _, _, taus), shapes in zip(engines, run(probe, engines)):
        assert shapes[0][2] == 0, (taus[-1], len(taus), shapes)


def test_the_measured_lists_keep_the_kernel(probe):
    """The lists whose launches were measured faster on this kernel still get it."""
    for taus in (log_taus(1, 500, 64), log_taus(1, 200, 64), log_taus(1, 100, 48), log_taus(1, 20, 20), log_taus(1, 1000, 64)):
        eb, *_ = run(probe, [(False, 32, taus[-1] + 64, 10 ** 6, 32, taus)])[0][0]
        assert eb in (16, 32), taus[-1]
