"""Integration where the two voxels of a thread part: the camera's own plane
(depth 0: quotients by zero, the voxel at the camera itself is 0 / 0), image
borders inside a block, pixels without depth, second observations, weights of
zero beside observed ones, and negative view angles' weights.  Every voxel must
equal the reference-precision oracle's, but for the voxel at the camera itself:
its pixel is the conversion of 0 / 0 to an integer, 0 on the GPU (the pixel
(0, 0)) and undefined on the CPU."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import golden_util as G
from tests.test_gpu_map import _session_for, dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# voxel size, truncation, camera translation, nearest depth
VIEWS = [(0.0625, 0.25, (0, 0, 0), 0.15), (0.0625, 0.5, (0, 0, 0.0625), 0.15), (0.03125, 0.125, (0.5, -0.25, -1), 0.15),
         (0.02, 0.06, (0.1, 0.2, 0.3), 0.3)]


@pytest.mark.parametrize("view", VIEWS, ids=[str(i) for i in range(len(VIEWS))])
def test_views(view):
    from fusion_b200 import system as S
    voxel, trunc, t, near = view
    m = G.meta()
    cfg = G.oracle_config(32)
    cfg.voxel_size, cfg.trunc_dist = voxel, trunc
    cfg.cx, cfg.cy = 64.0, 48.0
    M = O.Map(cfg)
    sess = _session_for(cfg)
    K = np.array([m["fx"], m["fy"], cfg.cx, cfg.cy], np.float32)
    H, W = G.load("pre_128x96.npz")["depth_in"].shape
    rng = np.random.default_rng(7)
    T = np.eye(4)
    T[:3, 3] = t
    for frame in range(3):
        depth = (near + 0.4 * rng.random((H, W)) ** 2 + 0.002 * np.arange(W)[None, :]).astype(np.float32)
        depth[rng.random((H, W)) < 0.1] = np.nan
        nm = rng.normal(size=(H, W, 4)).astype(np.float32)
        nm[..., :3] /= np.linalg.norm(nm[..., :3], axis=-1, keepdims=True)
        nm[..., 3] = 1.0
        rgb = rng.integers(0, 256, (H, W, 3), dtype=np.uint8)
        assert S.fuse_map_color(sess, dev(depth), dev(rgb), dev(nm), T, K) == M.fuse(depth, rgb, nm, T)
        e = M.entries()
        e = e[e[:, 3] >= 0]
        v = np.arange(512)
        pos = e[:, None, :3] * 8 + np.stack([v & 7, (v >> 3) & 7, v >> 6], -1)[None]
        camera = np.all(pos.astype(np.float32) * np.float32(voxel) == np.float32(t), axis=-1)
        (sdf_g, w_g, c_g), (sdf_o, w_o, c_o) = sess.blocks(e[:, 3]), M.voxels(e[:, 3])
        keep = ~camera.reshape(w_o.shape)
        assert np.count_nonzero(~keep) <= 1
        assert np.array_equal(w_g[keep], w_o[keep])
        assert np.array_equal(c_g[keep], c_o[keep])
        obs = keep & (w_o > 0)
        assert obs.any()
        assert np.array_equal(sdf_g[obs], sdf_o[obs].astype(np.float32))
    M.close()
    sess.close()
