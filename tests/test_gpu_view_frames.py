"""The model view of fused frames, whose z ranges are made with the visible
blocks in one pass, against the raycast entry on the same map and pose, which
makes them from the visible list: same tiles, same vertices and normals.
Alone and as a part of a fused batch step, in both forms, with a lost frame (no
depth) between; every size has to compare four frames of a moving camera."""
import numpy as np
import pytest

import rgbd_synth as synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _scene(cfg, step):
    """The first of eight scenes whose frames 1 to 3 are all tracked (a sparse
    first raycast can lose the camera): its frames, a frame without depth before
    the last one."""
    from fusion_b200 import Session
    for scene in range(8):
        p = synth.params(cfg.width, cfg.height, synth.session_seed(16, scene), fx=cfg.fx, fy=cfg.fy, cx=cfg.cx,
                         cy=cfg.cy, depth_scale=cfg.depth_scale)
        d, c, _ = synth.render(p, 0, 5)
        s = Session(cfg)
        ok = all([step(s, (d[k], c[k])).tracked for k in range(4)])
        s.close()
        if ok:
            return [(d[k], c[k]) for k in range(4)] + [(np.zeros_like(d[0]), c[4]), (d[4], c[4])]
    raise AssertionError("no scene is tracked")


@pytest.mark.parametrize("fused_step", [False, True])
@pytest.mark.parametrize("size,voxel,form", [((161, 121), 0.012, 0), ((640, 480), 0.006, 0), ((333, 251), 0.01, 1)])
def test_frames(size, voxel, form, fused_step):
    from fusion_b200 import Batch, Session, mixed_config
    from fusion_b200 import system as S
    w, h = size
    cfg = mixed_config(w, h, voxel, 8)
    cfg.form = form
    batch = Batch(mode=2)
    step = (lambda s, f: batch.step([s], [f])[0]) if fused_step else (lambda s, f: s.grab(*f))
    K = np.array([cfg.fx, cfg.fy, cfg.cx, cfg.cy], np.float32)
    frames = _scene(cfg, step)
    s, compared = Session(cfg), 0
    for k, f in enumerate(frames):
        r = step(s, f)
        assert bool(r.tracked) == (k != 4)
        if not r.tracked:
            continue
        lv, tiles = s.level(0, 0), s.stats()["no_tiles"]
        vm, nm = (torch.zeros((h, w, 4), dtype=torch.float32, device="cuda") for _ in range(2))
        assert S.raycast(s, vm, nm, s.pose(), K)
        torch.cuda.synchronize()
        assert tiles > 0 and s.stats()["no_tiles"] == tiles
        assert np.array_equal(vm.cpu().numpy(), lv["vmap"], equal_nan=True)
        assert np.array_equal(nm.cpu().numpy(), lv["nmap"], equal_nan=True)
        compared += k > 0
    assert compared == 4, compared
    s.close()
    batch.close()
