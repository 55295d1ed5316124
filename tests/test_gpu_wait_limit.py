"""The waits of the tracking kernel's blocks for one another end: with a limit
of no polls every wait for sums gives up, the kernel returns, and the frame is reported
as not tracked with FB_ERR_TIMEOUT and the last pose.  The frames that follow
are those of a session whose tracker failed that frame by its counts (a frame
without depth), bit for bit: alone, and beside another session in a batch step.
Sizes: every block with pixels at all levels and not, lists in shared and in
global memory; both forms."""
import time

import numpy as np
import pytest

import rgbd_synth as synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ERR_TIMEOUT = 0x80


def _limit(s, polls):
    return s.lib.fb_session_set_wait_limit(s.h, polls)


def _frames(cfg, seed, n):
    p = synth.params(cfg.width, cfg.height, synth.session_seed(15, seed), fx=cfg.fx, fy=cfg.fy, cx=cfg.cx, cy=cfg.cy,
                     depth_scale=cfg.depth_scale)
    d, c, _ = synth.render(p, 0, n)
    return [(d[k], c[k]) for k in range(n)]


@pytest.mark.parametrize("size,form", [((160, 120), 0), ((161, 123), 1), ((640, 480), 0), ((811, 607), 0)])
def test_alone(size, form):
    from fusion_b200 import Session, mixed_config
    cfg = mixed_config(*size, 0.010, 8)
    cfg.form = form
    frames = _frames(cfg, size[0], 6)
    s, other = Session(cfg), Session(cfg)
    for f in frames[:3]:
        s.grab(*f)
        last = other.grab(*f)
    assert last.tracked and not last.error_flags & ERR_TIMEOUT
    other.grab(np.zeros_like(frames[3][0]), frames[3][1])
    assert _limit(s, 0) == 0
    t = time.perf_counter()
    r = s.grab(*frames[3])
    assert time.perf_counter() - t < 1.0
    assert not r.tracked and r.error_flags & ERR_TIMEOUT
    assert list(r.pose) == list(last.pose)
    assert np.isnan(r.icp_error) and np.isnan(r.rgb_error) and r.icp_count == 0 and r.rgb_count == 0
    assert _limit(s, 1 << 18) == 0
    for f in frames[4:]:
        a, b = Session.result_dict(s.grab(*f)), Session.result_dict(other.grab(*f))
        assert a["tracked"]
        a["error_flags"] &= ~ERR_TIMEOUT   # sticky
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=True), (k, a[k], b[k])
    s.close()
    other.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_beside_another_session(mode):
    from fusion_b200 import Batch, Session, mixed_config
    cfg = mixed_config(323, 241, 0.012, 8)
    frames = [_frames(cfg, 50 + i, 6) for i in range(2)]
    ss, alone, batch = [Session(cfg) for _ in range(2)], Session(cfg), Batch(mode=mode)
    tracked = 0
    for k in range(6):
        assert _limit(ss[0], 0 if k == 3 else 1 << 18) == 0
        r = batch.step(ss, [f[k] for f in frames])
        assert bool(r[0].error_flags & ERR_TIMEOUT) == (k >= 3)
        assert not (k == 3 and r[0].tracked)
        a, b = Session.result_dict(r[1]), Session.result_dict(alone.grab(*frames[1][k]))
        tracked += a["tracked"]
        for key in a:
            assert np.array_equal(a[key], b[key], equal_nan=True), (k, key, a[key], b[key])
    assert tracked >= 4
    batch.close()
    for s in ss + [alone]:
        s.close()


def test_limits():
    from fusion_b200 import Session, mixed_config
    s = Session(mixed_config(160, 120, 0.02, 8))
    assert _limit(s, -1) == 1 and _limit(s, (1 << 18) + 1) == 1 and _limit(s, 1) == 0
    assert s.lib.fb_session_set_wait_limit(None, 1) == 1
    s.close()
