"""fb_mesh_scene writing fewer triangles than the map holds: the first
`max_triangles` of the whole mesh, at caps inside a block, at its ends and at
the ends of the mesh, in both forms; nothing beyond them is written."""
import ctypes

import numpy as np
import pytest

import rgbd_synth as synth

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form", [0, 1])
def test_caps(form):
    from fusion_b200 import Session, load, mixed_config
    cfg = mixed_config(160, 120, 0.02, 8)
    cfg.form = form
    p = synth.params(160, 120, synth.session_seed(13, 3), fx=cfg.fx, fy=cfg.fy, cx=cfg.cx, cy=cfg.cy,
                     depth_scale=cfg.depth_scale)
    d, c, _ = synth.render(p, 0, 2)
    s = Session(cfg)
    for k in range(2):
        s.grab(d[k], c[k])
    V, N, C = s.mesh()
    total = len(V) // 3
    assert total > 2000
    lib = load()
    for cap in (1, 2, 85, 86, 171, 700, total // 2, total - 1, total, total + 5):
        v = torch.full((3 * (total + 6), 3), -7.0, device="cuda")
        n = torch.full_like(v, -7.0)
        k = torch.full((3 * (total + 6) + 1, 3), 201, dtype=torch.uint8, device="cuda").view(-1)[1:1 + 9 * (total + 6)]
        torch.cuda.synchronize()
        count = ctypes.c_uint64()
        # the colours one byte off a word boundary
        assert lib.fb_mesh_scene(s.h, v.data_ptr(), n.data_ptr(), k.data_ptr(), cap, ctypes.byref(count), None) == 0
        assert count.value == total
        w = 3 * min(cap, total)
        assert np.array_equal(v[:w].cpu().numpy(), V[:w]) and bool((v[w:] == -7.0).all())
        assert np.array_equal(n[:w].cpu().numpy(), N[:w], equal_nan=True) and bool((n[w:] == -7.0).all())
        assert np.array_equal(k[:3 * w].cpu().numpy(), C[:w].reshape(-1)) and bool((k[3 * w:] == 201).all())
    s.close()
