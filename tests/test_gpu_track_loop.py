"""A session alone tracks a frame's iterations in one launch; sessions sharing
the GPU track them with a kernel per pass.  Both must give the same bits: the
one-launch form is run by Session.grab, the other by a fused batch step of one
session (mode 2), over sizes with one chunk of 256 pixels per block and
several, with remainders, with lists in shared and (from about 436 000 pixels)
in global memory, in both forms, with levels left out, and through frames
that fail at the first iteration (no depth)."""
import time

import numpy as np
import pytest

import rgbd_synth as synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASES = [
    # width, height, voxel size, form, iterations at levels 0, 1, 2
    (160, 120, 0.010, 0, (10, 5, 3)),
    (161, 123, 0.012, 1, (10, 5, 3)),
    (323, 241, 0.010, 0, (4, 0, 3)),
    (427, 319, 0.008, 1, (0, 5, 3)),
    (640, 480, 0.008, 0, (10, 5, 3)),
    (811, 607, 0.010, 0, (3, 2, 2)),
    (811, 607, 0.010, 1, (2, 0, 0)),
]


@pytest.mark.parametrize("case", CASES, ids=[f"{w}x{h}-form{f}-{i}" for w, h, _, f, i in CASES])
def test_one_launch_gives_the_passes_bits(case):
    from fusion_b200 import Batch, Session, mixed_config
    w, h, voxel, form, iters = case
    cfg = mixed_config(w, h, voxel, 8)
    cfg.form = form
    for l in range(3):
        cfg.iters[l] = iters[l]
    p = synth.params(w, h, synth.session_seed(12, w * 7 + h), fx=cfg.fx, fy=cfg.fy, cx=cfg.cx, cy=cfg.cy,
                     depth_scale=cfg.depth_scale)
    d, c, _ = synth.render(p, 0, 5)
    frames = [(d[k], c[k]) for k in range(4)] + [(np.zeros_like(d[0]), c[4]), (d[4], c[4])]
    alone, shared, batch = Session(cfg), Session(cfg), Batch(mode=2)
    tracked = 0
    for depth, rgb in frames:
        a = Session.result_dict(alone.grab(depth, rgb))
        b = Session.result_dict(batch.step([shared], [(depth, rgb)])[0])
        tracked += a["tracked"]
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=True), (k, a[k], b[k])
    assert tracked >= 3, tracked
    for l in range(3):
        va, vb = alone.level(0, l), shared.level(0, l)
        for k in va:
            assert np.array_equal(va[k], vb[k], equal_nan=va[k].dtype.kind == "f"), (l, k)
    alone.close()
    shared.close()


def test_failed_frames_end_at_once():
    """A frame that fails at the coarsest level ends for the blocks that only
    the finest level uses too: they must not wait for poses that never come
    (a wait that gives up takes some hundred milliseconds)."""
    from fusion_b200 import Session, mixed_config
    cfg = mixed_config(640, 480, 0.008, 8)
    p = synth.params(640, 480, synth.session_seed(12, 5), fx=cfg.fx, fy=cfg.fy, cx=cfg.cx, cy=cfg.cy,
                     depth_scale=cfg.depth_scale)
    d, c, _ = synth.render(p, 0, 3)
    s = Session(cfg)
    for k in range(3):
        s.grab(d[k], c[k])
    took = []
    for _ in range(5):
        t = time.perf_counter()
        r = s.grab(np.zeros_like(d[0]), c[0])
        took.append(time.perf_counter() - t)
        assert not r.tracked
    assert sorted(took)[2] < 0.05, took
    s.close()
