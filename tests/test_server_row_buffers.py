"""A served stream's FFT row buffer is a convenience: it never turns a stream away that the budget holds
without it, and all streams together stay within the budget."""
import threading

import numpy as np
import pytest

from cuda_multiddm_b200 import Engine, EngineConfig, Server, media

pytestmark = pytest.mark.gpu

SIDE, CHUNK = 256, 32
TAUS = media.log_taus(1, 20, 12)  # 84 ring slots and 12 sums per element; the row buffer: 32 frames
FRAME = 8 * sum((SIDE // s) ** 2 * s * (s // 2 + 1) for s in (256, 128))


def config():
    return EngineConfig(frame_width=SIDE, frame_height=SIDE, scales=[256, 128], taus=TAUS, lambdas=[4.0, 8.0, 16.0],
                        chunk_frames=CHUNK, lag_batch_frames=CHUNK)


def need(streams):
    """Device bytes of that many streams without row buffers, and a tenth of one stream more (annulus lists,
    tables, staged frames, results)."""
    return int(FRAME * (TAUS[-1] + 2 * CHUNK + len(TAUS)) * (streams + 0.1 * streams))


def alone(video):
    out = []
    with Engine(config()) as eng:
        for f in range(0, len(video), CHUNK):
            eng.submit(video[f:f + CHUNK])
            eng.finalize()
            out.append(eng.isf())
    return out


def test_row_buffers_make_room_for_streams():
    videos = [media.synth_video(3 + i, SIDE, SIDE, 3 * CHUNK, 80, step_var=1.0) for i in range(2)]
    want = [alone(v) for v in videos]
    with Server(hbm_budget_bytes=need(2)) as srv:
        ids = [srv.add_stream(config())]
        first = srv.stats()["device_bytes"]
        assert first > need(1) * 10 // 11 + 16 * FRAME  # with its row buffer
        srv.submit(ids[0], videos[0][:CHUNK])
        assert srv.step() == 1  # queued work uses the buffer when it is taken back
        ids.append(srv.add_stream(config()))
        assert ids[1] is not None
        assert srv.stats()["device_bytes"] <= need(2)
        assert srv.add_stream(config()) is None
        srv.submit(ids[1], videos[1][:CHUNK])
        for k in (1, 2):
            for sid, v in zip(ids, videos):
                srv.submit(sid, v[k * CHUNK:(k + 1) * CHUNK])
        got = {sid: [] for sid in ids}
        for _ in range(3):
            srv.step()
            srv.wait()
            for sid in ids:
                while (r := srv.poll(sid)) is not None:
                    got[sid].append(r[1])
        for sid, w in zip(ids, want):
            assert len(got[sid]) == 3 and all(np.array_equal(a, b) for a, b in zip(got[sid], w))
        srv.remove_stream(ids[1])
        srv.wait()
        srv.remove_stream(ids[0])
        srv.wait()
        sid = srv.add_stream(config())  # room again: with a row buffer
        assert srv.stats()["device_bytes"] == first
        srv.remove_stream(sid)


def test_streams_added_at_once_stay_within_the_budget():
    with Server(hbm_budget_bytes=need(3)) as srv:
        ids = [None] * 3

        def add(i):
            ids[i] = srv.add_stream(config())

        threads = [threading.Thread(target=add, args=(i,)) for i in range(3)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert None not in ids
        assert srv.stats()["device_bytes"] <= need(3)
