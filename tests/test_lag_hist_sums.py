"""The resident-history lag kernel's sums over the engine's own spectra (read back after every call):
within 1e-5 of the same sums in float64, and the bits of the ring kernel (the static entry point) given
the same spectra in the same batches. Covers the first frames (masks), fused runs, launches of two batches,
batches cut at the end of a call, frame counts without an instance, and every shape of the kernel.

The bound: a launch sums up to 32 pairs in FP32. A difference rounds once and its square and sums at most
34 times, all terms positive, so a launch is within 36 * 2^-24 = 2.1e-6 of itself and the Kahan sum over
launches adds 2 * 2^-24; 1e-5 of the sum holds for every element by itself."""
import ctypes as C

import numpy as np
import pytest
import torch

from cuda_multiddm_b200 import Engine, EngineConfig, lib, media

pytestmark = pytest.mark.gpu

RUNS = list(range(1, 14)) + [17, 18, 19, 20, 21, 33, 60, 61, 62, 63, 90]


def batches(calls, chunk):
    """Frame ranges the engine pairs at once: chunks of 32 frames and more are paired piece by piece within a
    call, smaller ones in batches of 32 across calls, the rest when a result is read."""
    out, n0, n = [], 0, 0
    for c in calls:
        n += c
        if chunk >= 32:
            while n0 < n:
                out.append((n0, min(32, n - n0)))
                n0 += out[-1][1]
        else:
            while n - n0 >= 32:
                out.append((n0, 32))
                n0 += 32
    if n0 < n:
        out.append((n0, n - n0))
    return out


@pytest.mark.parametrize("side,scales,taus,chunk,calls", [
    (64, [64, 32], media.log_taus(1, 40, 12), 7, (1, 6, 33, 20)),
    (64, [64, 16], RUNS, 32, (31, 64, 3, 90, 40)),
    (256, [256, 16], media.log_taus(1, 260, 64), 32, (40, 300, 5)),
    (512, [512, 256, 128, 64], media.log_taus(1, 90, 40), 30, (150, 64, 31)),
    (512, [512, 256, 128, 64], RUNS, 32, (150, 64, 95)),
    (256, [256, 128], media.log_taus(1, 620, 64), 17, (600, 130)),
    (512, [512, 256], media.log_taus(1, 300, 64), 32, (310, 64, 32, 9)),  # launches that ask for more shared memory
    (512, [512, 256], list(range(1, 21)), 30, (75, 40)),                  # than their tables need
])
def test_sums_match_float64_and_the_ring_kernel(side, scales, taus, chunk, calls):
    rng = np.random.default_rng(side + chunk)
    n = sum(calls)
    frames = rng.integers(0, 256, (n, side, side), dtype=np.uint8)
    with Engine(EngineConfig(frame_width=side, frame_height=side, scales=scales, taus=taus, lambdas=[4.0, 8.0],
                             chunk_frames=chunk)) as eng:
        assert max(calls) <= eng.info().ring_slots
        spectra, done = [], 0
        for c in calls:
            eng.submit(frames[done:done + c])
            spectra += [torch.from_numpy(eng.spectrum(f)).cuda() for f in range(done, done + c)]
            done += c
        got = torch.from_numpy(eng.accumulators()).cuda()
    ring = torch.view_as_real(torch.stack(spectra)).contiguous()  # [n, E, 2]
    E = ring.shape[1]
    acc = torch.zeros((len(taus), E, 2), device="cuda")
    order = sorted(taus, reverse=True)  # windows ascend
    for n0, c in batches(calls, chunk):
        a = np.arange(n0, n0 + c, dtype=np.int32)
        b = np.stack([np.where(a - t >= 0, a - t, -1) for t in order]).astype(np.int32)
        st = lib().ddm_lag_accumulate_static(C.c_void_p(ring.data_ptr()), n, E, C.c_void_p(acc.data_ptr()), a.ctypes.data,
                                             c, b.ctypes.data, len(taus), None)
        assert st == 0, lib().ddm_last_error()
    acc = acc.double().flip(0)
    ring_kernel = acc[..., 0] - acc[..., 1]
    for i, tau in enumerate(taus):
        want = torch.zeros(E, dtype=torch.float64, device="cuda")
        for t in range(tau, n):
            want += (ring[t].double() - ring[t - tau].double()).square().sum(-1)
        assert bool(((got[i] - want).abs() <= 1e-5 * want).all()), tau
    assert torch.equal(got, ring_kernel)
