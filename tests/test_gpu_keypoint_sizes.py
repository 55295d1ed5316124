"""Key points at sizes whose octaves have remainders (all octaves run in one
launch over the largest one's grid) and near the image's edge, where the Haar
boxes are clipped: positions, angles and descriptors against the numpy
restatement, as in test_gpu_keypoints, which derives the tolerances."""
import numpy as np
import pytest

import rgbd_synth as synth
from oracle import keypoints as OK

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size", [(161, 121), (257, 193), (400, 131)])
def test_sizes(size):
    from fusion_b200 import Session, mixed_config
    from oracle import oracle as O
    w, h = size
    cfg = mixed_config(w, h, 0.01, 8)
    p = synth.params(w, h, synth.session_seed(15, w), fx=cfg.fx, fy=cfg.fy, cx=cfg.cx, cy=cfg.cy,
                     depth_scale=cfg.depth_scale)
    d, c, _ = synth.render(p, 0, 1)
    s = Session(cfg)
    s.set_keypoints(True)
    s.grab(d[0], c[0])
    g, lv = s.keypoints(0), s.level(0, 0)
    s.close()
    depth = np.ascontiguousarray(lv["depth"], np.float32)
    nm = O.nmap(O.vmap(depth, cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.depth_cutoff, 32), 32).astype(np.float32)
    kp_all, desc_all = OK.detect(lv["image"])
    kp, _, _, desc = OK.backproject(kp_all, desc_all, depth, nm, cfg.fx, cfg.fy, cfg.cx, cfg.cy, cfg.depth_cutoff)
    n_g, n_o = len(g["kp"]), len(kp)
    assert n_o >= 20 and abs(n_g - n_o) <= max(1, 0.02 * n_o), (n_g, n_o)
    good = 0
    for i in range(n_g):
        dd = np.abs(kp[:, :2] - g["kp"][i, :2]).max(axis=1)
        j = int(np.argmin(dd))
        if dd[j] > 1e-3:
            continue
        turn = abs((kp[j, 3] - g["kp"][i, 3] + np.pi) % (2 * np.pi) - np.pi)
        good += turn < 1e-3 and np.abs(desc[j] - g["desc"][i]).max() < 1e-3
    assert good >= 0.95 * n_o, (good, n_o)
