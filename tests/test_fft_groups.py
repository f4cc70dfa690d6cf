"""ddm_config.fft_group_frames is the number of frames of an FFT launch, also where that is more than 256 MB
of spectra hold: what ddm_get_info reports is what runs, and the results do not depend on it."""
import numpy as np
import pytest

from cuda_multiddm_b200 import Engine, EngineConfig, media

pytestmark = pytest.mark.gpu


def test_groups_above_256_mb_run_as_asked():
    side, scales, taus = 1024, [1024, 512, 256, 128, 64, 32, 16], media.log_taus(1, 20, 10)
    frame = 8 * sum((side // s) ** 2 * s * (s // 2 + 1) for s in scales)
    assert (256 << 20) // frame == 8
    video = media.synth_video(5, side, side, 32, 400, step_var=1.0)
    launches, isf = {}, {}
    for group in (0, 8, 16, 32):
        with Engine(EngineConfig(frame_width=side, frame_height=side, scales=scales, taus=taus, lambdas=[4.0, 8.0],
                                 chunk_frames=32, fft_group_frames=group)) as eng:
            eng.submit(video)
            eng.finalize()
            assert eng.info().fft_group_frames == group
            launches[group], isf[group] = eng.info().kernel_launches, eng.isf()
    assert launches[8] == launches[0]
    assert launches[0] - launches[16] == 2 * (4 - 2) and launches[0] - launches[32] == 2 * (4 - 1)  # two passes a group
    assert all(np.array_equal(v, isf[0]) for v in isf.values())
