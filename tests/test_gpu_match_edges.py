"""fb_match_descriptors at the edges of its tiles and clusters: one query and
train, remainders of 8 and 32 queries and of 256 trains, sizes of both shapes
and of several cluster sizes, equal distances (the lower index first), trains
with infinities and NaN (never a match), descriptors off a 16-byte boundary.
Against distances in 64 bits; a chain of 64 FMAs of values below 4 is within
64 * 2^-24 of them relative to the sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SIZES = [(1, 1), (1, 2), (7, 3), (8, 255), (9, 256), (33, 257), (65, 513), (31, 2049), (700, 1500), (1201, 2600)]


def _unaligned(a):
    flat = torch.zeros(a.size + 1, dtype=torch.float32, device="cuda")
    flat[1:] = torch.from_numpy(a.reshape(-1)).cuda()
    return flat[1:].view(a.shape)


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("size", SIZES, ids=[f"{q}x{t}" for q, t in SIZES])
def test_sizes(size, aligned):
    from fusion_b200.system import match_descriptors
    nq, nt = size
    rng = np.random.default_rng(nq * 10007 + nt)
    t = rng.uniform(-1, 1, (nt, 64)).astype(np.float32)
    q = rng.uniform(-1, 1, (nq, 64)).astype(np.float32)
    for i in range(0, nt - 1, 5):            # equal trains: a tie at every distance
        t[nt - 1 - i] = t[i]
    if nt > 4:
        t[2, 7], t[3, 0] = np.inf, np.nan    # an infinite and a NaN distance
    for i in range(0, nq, 3):                # some queries are a train: distance zero, twice where it has a twin
        q[i] = t[min(5, nt - 1)]
    put = (lambda a: torch.from_numpy(a).cuda()) if aligned else _unaligned
    best, dist = (x.cpu().numpy() for x in match_descriptors(put(q), put(t)))
    for i in range(nq):
        with np.errstate(invalid="ignore"):
            d = np.sqrt(np.square(q[i].astype(np.float64) - t).sum(1))
        ok = np.nonzero(np.isfinite(d))[0]
        order = ok[np.lexsort((ok, d[ok]))][:2]
        for k in range(2):
            if k < len(order):
                assert best[i, k] == order[k], (i, k, best[i], order)
                assert abs(dist[i, k] - d[order[k]]) <= 64 * 2.0 ** -24 * d[order[k]], (i, k)
            else:
                assert best[i, k] == -1 and np.isinf(dist[i, k]), (i, k, best[i], dist[i])
