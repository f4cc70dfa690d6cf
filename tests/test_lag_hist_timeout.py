"""The resident-history lag kernel's bounded waits (8 taus and more): a stage barrier that expects one
arrival more than the producer makes (host-side fault injection) makes the consumers' waits run out after
a short limit; every warp leaves together, the kernel returns a status, finalize reports it, and the next
engine computes correct results. One list per shape of the kernel: whole blocks in several row buffers,
register-frame buffers with blocks of 32 and of 16 elements, one CTA per SM."""
import numpy as np
import pytest

from cuda_multiddm_b200 import DDMError, Engine, EngineConfig, media
from cuda_multiddm_b200._lib import FAULT_LAG_WAIT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taus,frames", [
    (list(range(1, 21)), 60), (media.log_taus(1, 110, 24), 150), (media.log_taus(1, 300, 40), 64),
    (media.log_taus(1, 600, 64), 64)])
def test_wait_timeout_is_reported_and_the_device_stays_usable(taus, frames):
    side, scales, lambdas = 64, [64, 32], [4.0, 8.0, 16.0]
    video = media.synth_video(5, side, side, frames, 20, step_var=1.0)
    cfg = EngineConfig(frame_width=side, frame_height=side, scales=scales, taus=taus, lambdas=lambdas, chunk_frames=32)
    with Engine(cfg) as eng:
        eng.submit(video)
        eng.finalize()
        want = eng.isf()
    with Engine(cfg) as eng:
        eng.set_wait_limit(2_000_000)  # about 1 ms of SM clocks
        eng.inject_fault(FAULT_LAG_WAIT)
        eng.submit(video)
        with pytest.raises(DDMError) as info:
            eng.finalize()
        assert info.value.status == 2 and "timed out" in str(info.value)
    with Engine(cfg) as eng:
        eng.submit(video)
        eng.finalize()
        assert np.array_equal(eng.isf(), want)
