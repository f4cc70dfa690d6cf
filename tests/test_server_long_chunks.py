"""Served chunks of more than 32 frames queue several lag launches of one stream; they update the
same sums and must run one after another (both lag kernels: 12 and 5 taus)."""
import numpy as np
import pytest

from cuda_multiddm_b200 import Engine, EngineConfig, Server, media

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taus", [media.log_taus(1, 40, 12), [1, 2, 3, 5, 8]])
def test_long_chunks_equal_the_engine_alone(taus):
    C, chunks, side = 64, 3, 128
    cfg = dict(frame_width=side, frame_height=side, scales=[128, 32], taus=taus, lambdas=[4.0, 8.0, 16.0],
               chunk_frames=C, lag_batch_frames=32)
    video = media.synth_video(9, side, side, C * chunks, 80, step_var=1.0)
    want = []
    with Engine(EngineConfig(**cfg)) as eng:
        for k in range(chunks):
            for f in range(0, C, 32):  # the pieces a served chunk is cut into
                eng.submit(video[k * C + f:k * C + min(f + 32, C)])
            eng.finalize()
            want.append(eng.isf())
    with Server() as srv:
        sid = srv.add_stream(EngineConfig(**cfg))
        for k in range(chunks):
            srv.submit(sid, video[k * C:(k + 1) * C])
            srv.step()
            srv.wait()
            _, isf = srv.poll(sid)
            assert np.array_equal(isf, want[k])
