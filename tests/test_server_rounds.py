"""Served chunks of any length, and steps queued one after another without a wait: the same results, bit
for bit, as the engine alone that is given the same frames piece by piece. A chunk longer than two pieces
(min(chunk_frames, 32) frames each) used to overwrite partners that its own lag launches still had to
read, and two steps with chunks of two pieces raced on the ring."""
import numpy as np
import pytest

from cuda_multiddm_b200 import Engine, EngineConfig, Server, media

pytestmark = pytest.mark.gpu

SIDE, STEPS = 128, 4
LISTS = (media.log_taus(1, 70, 14), [1, 2, 3, 5, 70])  # both lag kernels


def config(chunk, taus):
    return EngineConfig(frame_width=SIDE, frame_height=SIDE, scales=[128, 32], taus=taus, lambdas=[4.0, 8.0, 16.0],
                        chunk_frames=chunk, lag_batch_frames=min(chunk, 32))


def alone(cfg, video, count):
    """The ISF after every `count` frames."""
    piece, out = min(cfg.chunk_frames, 32), []
    with Engine(cfg) as eng:
        for k in range(0, len(video), count):
            for f in range(k, k + count, piece):
                eng.submit(video[f:min(f + piece, k + count)])
            eng.finalize()
            out.append(eng.isf())
    return out


@pytest.mark.parametrize("taus", LISTS)
@pytest.mark.parametrize("chunk,count", [(32, 64), (20, 60), (64, 65), (32, 200), (10, 33)])
@pytest.mark.parametrize("wait", [False, True])
def test_chunks_of_any_length_equal_the_engine_alone(taus, chunk, count, wait):
    cfg = config(chunk, taus)
    video = media.synth_video(9, SIDE, SIDE, count * STEPS, 80, step_var=1.0)
    want = alone(cfg, video, count)
    with Server(results_per_stream=STEPS) as srv:
        sid = srv.add_stream(cfg)
        for k in range(STEPS):
            srv.submit(sid, video[k * count:(k + 1) * count])
            assert srv.step() == 1
            if wait:
                srv.wait()
        srv.wait()
        for k in range(STEPS):
            res, isf = srv.poll(sid)
            assert res["chunk_index"] == k and res["frames"] == (k + 1) * count
            assert np.array_equal(isf, want[k])


def test_streams_of_different_chunk_lengths_share_steps():
    cfgs = [config(32, LISTS[0]), config(20, LISTS[0]), config(30, LISTS[1])]
    counts = [20, 130, 64]
    videos = [media.synth_video(3 + i, SIDE, SIDE, n * STEPS, 80, step_var=1.0) for i, n in enumerate(counts)]
    want = [alone(c, v, n) for c, v, n in zip(cfgs, videos, counts)]
    with Server(results_per_stream=STEPS) as srv:
        ids = [srv.add_stream(c) for c in cfgs]
        for k in range(STEPS):
            for sid, v, n in zip(ids, videos, counts):
                srv.submit(sid, v[k * n:(k + 1) * n])
            assert srv.step() == len(ids)
        srv.wait()
        for sid, w in zip(ids, want):
            for k in range(STEPS):
                assert np.array_equal(srv.poll(sid)[1], w[k])
