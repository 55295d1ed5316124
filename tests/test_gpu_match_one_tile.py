"""fb_match_descriptors with trains of one tile, where the kernel stages and
works on the parts of 128 trains there are: one train, both sides of a
part's end, and more query groups than are resident at once.  Against
distances in 64 bits; a chain of 64 FMAs of values below 4 is within 64 * 2^-24
of them relative to the sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("size", [(600, 1), (33, 127), (601, 128), (33, 129), (9001, 130), (5003, 64), (600, 256)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_one_tile(size):
    from fusion_b200.system import match_descriptors
    nq, nt = size
    rng = np.random.default_rng(nq * 10007 + nt)
    t = rng.uniform(-1, 1, (nt, 64)).astype(np.float32)
    q = rng.uniform(-1, 1, (nq, 64)).astype(np.float32)
    if nt > 2:
        t[nt - 1] = t[0]   # a tie: the lower index first
        q[nq // 2] = t[0]
    best, dist = (x.cpu().numpy() for x in match_descriptors(torch.from_numpy(q).cuda(), torch.from_numpy(t).cuda()))
    d = np.sqrt(np.maximum(((q[:, None, :].astype(np.float64) - t[None]) ** 2).sum(2), 0))
    order = np.argsort(d, axis=1, kind="stable")[:, :2]
    for k in range(2):
        if k < nt:
            assert np.array_equal(best[:, k], order[:, k])
            want = np.take_along_axis(d, order, 1)[:, k]
            assert (np.abs(dist[:, k] - want) <= 64 * 2.0 ** -24 * want).all()
        else:
            assert (best[:, k] == -1).all() and np.isinf(dist[:, k]).all()
