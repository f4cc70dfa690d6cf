"""Short lags of very large frames stay on the ring kernel (CPU, through tests/hist_rule_probe.cu), and such an
engine gives the reference sums (GPU)."""
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "cuda_multiddm_b200" / "csrc"
SRC = ROOT / "tests" / "hist_rule_probe.cu"
PROBE = ROOT / "tests" / "_build" / "hist_rule_probe"


def elements(side, *scales):
    return sum((side // s) ** 2 * s * (s // 2 + 1) for s in scales)


def test_rule():
    deps = [SRC] + [CSRC / f for f in ("lag_hist_host.hpp", "lag_hist.cuh", "lag_host.hpp", "lag.cuh", "layout.cuh")]
    if not PROBE.exists() or PROBE.stat().st_mtime < max(p.stat().st_mtime for p in deps):
        PROBE.parent.mkdir(parents=True, exist_ok=True)
        tmp = PROBE.with_name(f"{PROBE.name}.{os.getpid()}")
        subprocess.run(["nvcc", "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC),
                        str(SRC), "-o", str(tmp)], check=True)
        os.replace(tmp, PROBE)
    big = elements(2048, 2048, 1024)
    cases = {(big, 2, 39, 32): 1, (big, 2, 40, 32): 0, (big, 2, 20, 30): 1, (big, 2, 20, 25): 0, (big, 2, 20, 64): 1,
             (big, 2, 20, 48): 1, (big, 2, 20, 45): 0, (big, 2, 20, 16): 1, (elements(4096, 4096), 1, 20, 32): 1,
             (elements(2048, 2048), 1, 20, 32): 0, (elements(2048, 2048, 1024, 512, 256), 4, 20, 32): 0,
             (elements(256, 256), 1, 20, 30): 0}
    text = "".join(" ".join(map(str, c)) + "\n" for c in cases)
    out = subprocess.run([str(PROBE)], input=text, capture_output=True, text=True, check=True).stdout.split()
    assert [int(v) for v in out] == list(cases.values())


@pytest.mark.gpu
def test_sums_on_either_side_of_the_rule():
    from cuda_multiddm_b200 import Engine, EngineConfig, media
    side, scales, taus = 2048, [2048, 1024], list(range(1, 13)) + [20]
    video = media.synth_video(3, side, side, 40, 300, step_var=1.0)
    isf = []
    for chunk in (32, 25):  # ring kernel; resident history
        with Engine(EngineConfig(frame_width=side, frame_height=side, scales=scales, taus=taus, lambdas=[4.0, 32.0, 300.0],
                                 chunk_frames=chunk, lag_batch_frames=20)) as eng:
            for f in range(0, 40, 20):  # the same batches either way
                eng.submit(video[f:f + 20])
            eng.finalize()
            isf.append(eng.isf())
    assert np.array_equal(*isf)
