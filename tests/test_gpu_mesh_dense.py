"""Mesh extraction of noise: maps fused from random depths, where most cubes of
a block hold surface, cases of every kind meet missing, unobserved and saturated
voxels in the same row, and blocks hold more vertices than one round of a CTA
writes.  Against the oracle's restatement on the session's map, bit for bit."""
import numpy as np
import pytest

from fusion_b200 import system as S
from tests.test_gpu_mesh import _report, _rows, _session_map, _sorted, dev

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("spread,holes", [(0.02, 0.0), (0.3, 0.02), (0.3, 0.3)])
def test_noise(form, spread, holes):
    from fusion_b200 import Session, mixed_config
    from fusion_b200.system import mesh_case_table
    W, H, voxel = 160, 120, 0.02
    cfg = mixed_config(W, H, voxel, 8)
    cfg.form = form
    s = Session(cfg)
    K = np.array([cfg.fx, cfg.fy, cfg.cx, cfg.cy], np.float32)
    rng = np.random.default_rng(3)
    for frame in range(2):
        depth = (0.8 + spread * rng.random((H, W))).astype(np.float32)
        depth[rng.random((H, W)) < holes] = np.nan
        nm = np.tile(np.float32([0, 0, 1, 1]), (H, W, 1))
        rgb = rng.integers(0, 256, (H, W, 3), dtype=np.uint8)
        S.fuse_map_color(s, dev(depth), dev(rgb), dev(nm), np.eye(4), K)
    V, N, C = s.mesh()
    tri, cnt = mesh_case_table()
    M = _session_map(s)
    Vo, No, Co = M.mesh(tri, cnt, fused=1)
    assert len(Vo) == len(V) > 3000
    a, b = _rows(*_sorted(Vo, No, Co)), _rows(*_sorted(V, N, C))
    assert np.array_equal(a, b), _report(a, b)
    M.close()
    s.close()
