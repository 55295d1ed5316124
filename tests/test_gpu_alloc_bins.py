"""Block allocation and the frame's z ranges over table sizes where the
insertion's bins behave differently: one bucket for all blocks, buckets far
fewer than blocks (long chains inside a bin), a size that is no power of two,
one bucket per bin and several, pools and excess lists that just suffice and
just do not (the sequential path).  Against the reference-precision oracle,
two frames each: every slot, link, counter and visible block, and the z-range
images the raycast starts from."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import golden_util as G
from tests.test_gpu_map import _compare_maps, _session_for, dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# buckets, excess slots, blocks; frame A allocates about 540 blocks, A and B together about 640
TABLES = [(1, 4096, 4096), (7, 4096, 4096), (64, 1024, 2048), (1000, 1000, 1000), (4096, 512, 1024), (4097, 512, 1024),
          (12289, 512, 1024), (1 << 18, 64, 1024), (64, 300, 4096), (1 << 14, 1 << 12, 560)]


@pytest.mark.parametrize("table", TABLES, ids=[f"{b}-{e}-{n}" for b, e, n in TABLES])
def test_tables(table):
    from fusion_b200 import system as S
    m = G.meta()
    pre, st, fz = G.load("pre_128x96.npz"), G.load("steps_128x96.npz"), G.load("fuse_128x96.npz")
    cfg = G.oracle_config(32)
    cfg.num_buckets, cfg.num_excess, cfg.num_blocks = table
    M = O.Map(cfg)
    sess = _session_for(cfg)
    K = np.array([m["fx"], m["fy"], m["cx"], m["cy"]], np.float32)
    H, W = pre["depth_in"].shape
    for depth, rgb, nm, T in ((pre["depth_in"], pre["rgb_in"], pre["nmap0"], np.eye(4)),
                              (st["depth_in"], st["rgb_in"], st["B_nmap0"], fz["b_pose"])):
        raw, _ = O.filter_depth(depth, m["depth_scale"], m["depth_cutoff"], 32)
        n_o = M.fuse(raw, rgb, nm, T)
        n_g = S.fuse_map_color(sess, dev(raw), dev(rgb), dev(nm), T, K)
        assert n_g == n_o
        assert sorted(sess.visible().tolist()) == sorted(M.visible().tolist())
        _compare_maps(sess, M)
        vm = torch.full((H, W, 4), float("nan"), device="cuda")
        nmp = torch.full((H, W, 4), float("nan"), device="cuda")
        assert S.raycast(sess, vm, nmp, T, K)
        vo, _, zmin, zmax, tiles = M.raycast(T)
        torch.cuda.synchronize()
        assert sess.stats()["no_tiles"] == tiles
        assert np.array_equal(np.isnan(vm.cpu().numpy()[..., 0]), np.isnan(vo[..., 0]))
    M.close()
    sess.close()


def test_frames_equal_separate_stages():
    """A fused frame makes its z ranges with the visible blocks; the raycast
    entry makes them from the list.  Both give the same model view."""
    import rgbd_synth as synth
    from fusion_b200 import Session, mixed_config
    from fusion_b200 import system as S
    for w, h, voxel in ((161, 121, 0.02), (640, 480, 0.006), (333, 251, 0.01)):
        cfg = mixed_config(w, h, voxel, 8)
        p = synth.params(w, h, synth.session_seed(14, w), fx=cfg.fx, fy=cfg.fy, cx=cfg.cx, cy=cfg.cy,
                         depth_scale=cfg.depth_scale)
        d, c, _ = synth.render(p, 0, 3)
        s = Session(cfg)
        for k in range(3):
            r = s.grab(d[k], c[k])
            if not r.tracked:
                continue
            lv = s.level(0, 0)
            tiles = s.stats()["no_tiles"]
            vm, nmp = (torch.zeros((h, w, 4), dtype=torch.float32, device="cuda") for _ in range(2))
            K = np.array([cfg.fx, cfg.fy, cfg.cx, cfg.cy], np.float32)
            assert S.raycast(s, vm, nmp, s.pose(), K)
            torch.cuda.synchronize()
            assert s.stats()["no_tiles"] == tiles
            assert np.array_equal(vm.cpu().numpy(), lv["vmap"], equal_nan=True)
            assert np.array_equal(nmp.cpu().numpy(), lv["nmap"], equal_nan=True)
        s.close()
