"""The FFT column pass takes the frames of a few columns together only for large frames; spectra and results
have the same bits in either order, and without the row pass's own buffer (a budget that leaves it out)."""
import numpy as np
import pytest

from cuda_multiddm_b200 import Engine, EngineConfig, media

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,scales,frames", [
    (2048, [2048, 1024, 512, 256], 9),  # 67 MB a frame: frames first, groups of three
    (2048, [2048, 512], 10),            # 34 MB: frame by frame
    (512, [512, 64], 33),
])
def test_spectra_do_not_depend_on_the_order(side, scales, frames):
    taus = [1, 2, 3, 4, 5, 6, 7, 8]
    video = media.synth_video(7, side, side, frames, 300, step_var=1.0)
    cfg = dict(frame_width=side, frame_height=side, scales=scales, taus=taus, lambdas=[4.0, 8.0, 16.0], chunk_frames=frames)

    def run(budget):
        with Engine(EngineConfig(**cfg, hbm_budget_bytes=budget)) as eng:
            eng.submit(video)
            eng.finalize()
            return eng.isf(), [eng.spectrum(f) for f in (0, 1, frames // 2, frames - 1)], eng.info().device_bytes

    isf, spectra, full = run(0)
    frame = 8 * sum((side // s) ** 2 * s * (s // 2 + 1) for s in scales)
    isf2, spectra2, less = run(full - frame)
    assert less < full  # without the buffer
    assert np.array_equal(isf, isf2)
    assert all(np.array_equal(a, b) for a, b in zip(spectra, spectra2))
