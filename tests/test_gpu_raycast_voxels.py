"""The raycast's trilinear reads where their voxels are awkward: surfaces on
both sides of the world's origin (coordinates truncate toward zero), rays whose
x or y coordinate is the float just above -1 voxel for a whole image column or
row (p - 1 and p + 1 then round to other voxels than their neighbours', the
normal's general form), and maps far from the origin.  Against the
reference-precision oracle on the same map: the same pixels hit, vertices
within 1e-5 m and normals within 1e-4, the bounds of the map's own test."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import golden_util as G
from tests.test_gpu_map import _session_for, dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

VOXEL = 1.0 / 64
EDGE = (-1.0 + 2.0 ** -24) * VOXEL      # a float; divided by the voxel size, the float next to -1
VIEWS = [(0, 0, 0), (EDGE, 0, 0), (0, EDGE, 0), (EDGE, EDGE, EDGE), (-0.37, 0.21, -1.13), (-37.2, 11.3, 5.9)]


@pytest.mark.parametrize("t", VIEWS, ids=[str(i) for i in range(len(VIEWS))])
def test_views(t):
    from fusion_b200 import system as S
    m = G.meta()
    pre = G.load("pre_128x96.npz")
    cfg = G.oracle_config(32)
    cfg.voxel_size = VOXEL
    cfg.trunc_dist = 4 * VOXEL
    cfg.cx, cfg.cy = 64.0, 48.0         # the optical axis is the ray of a pixel: its x and y stay the camera's
    M = O.Map(cfg)
    sess = _session_for(cfg)
    K = np.array([m["fx"], m["fy"], cfg.cx, cfg.cy], np.float32)
    T = np.eye(4)
    T[:3, 3] = t
    raw, _ = O.filter_depth(pre["depth_in"], m["depth_scale"], m["depth_cutoff"], 32)
    assert S.fuse_map_color(sess, dev(raw), dev(pre["rgb_in"]), dev(pre["nmap0"]), T, K) == \
        M.fuse(raw, pre["rgb_in"], pre["nmap0"], T)
    H, W = raw.shape
    vm = torch.full((H, W, 4), float("nan"), device="cuda")
    nm = torch.full((H, W, 4), float("nan"), device="cuda")
    assert S.raycast(sess, vm, nm, T, K)
    vo, no, _, _, _ = M.raycast(T)
    torch.cuda.synchronize()
    gv, gn = vm.cpu().numpy(), nm.cpu().numpy()
    hit = ~np.isnan(vo[..., 0])
    assert hit.any()
    assert np.array_equal(~np.isnan(gv[..., 0]), hit)
    assert np.abs(gv[hit] - vo[hit]).max() <= 1e-5
    assert np.abs(gn[hit] - no[hit]).max() <= 1e-4
    M.close()
    sess.close()
