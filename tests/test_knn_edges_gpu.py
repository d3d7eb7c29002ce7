"""pm_knn and pm_knn_noalloc where a query's set is odd: records that are NaN
in some coordinate beside the query, queries at infinity or NaN, an infinite
radius, more records at one place than a warp's registers hold. The result is
a brute-force sort by (squared distance, index), NaN distances left out, bit
for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402

pytestmark = pytest.mark.gpu


def records(kind, n, rs):
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5], size=(n, 3))
    if kind == "nan_axis":      # two of three records lack one coordinate
        for a in range(2):
            p[a::3, a] = np.nan
    elif kind == "nan_most":    # nine of ten lack all three
        p[np.arange(n) % 10 != 0, :3] = np.nan
    elif kind == "infinite":    # beside queries at infinity: no distance, and boxes without end
        p[::5, 0], p[1::7, 1], p[2::9, :3] = -np.inf, np.inf, -np.inf
    elif kind == "piles":       # places of 1, 20, 400 and 1,000 records
        for i, m in enumerate((1000, 400, 20)):
            p[i: i + 4 * m: 4, :3] = np.float32([0.1 * i, 0.5, 0.0])
    return p


def queries(kind, p, rs):
    q = np.zeros((96, 4), np.float32)
    q[:, :3] = rs.uniform([-0.6, -0.1, -0.6], [0.6, 1.1, 0.6], size=(96, 3))
    ok = np.isfinite(p[:, :3]).all(1)
    q[:48, :3] = p[rs.choice(np.flatnonzero(ok), 48), :3]
    if kind == "odd":
        q[0, 0] = np.nan
        q[1, :3] = np.nan
        q[2, 1] = np.inf
        q[3, :3] = -np.inf
        q[4, :3] = 1e30
        q[5, 2] = -3e19
    return q


def brute(p, q, k, radius):
    with np.errstate(all="ignore"):
        r2 = np.float32(radius) * np.float32(radius)
        idx = np.full((len(q), k), 0xFFFFFFFF, np.uint32)
        d2 = np.full((len(q), k), r2, np.float32)
        for i, x in enumerate(q):
            d = p[:, :3] - x[:3]
            s = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
            c = np.flatnonzero(s <= r2)
            c = c[np.lexsort((c, s[c]))][:k]
            idx[i, : len(c)] = c
            d2[i, : len(c)] = s[c]
    return idx, d2


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("k,radius", [(1, 0.3), (10, 0.4), (33, 2.0), (128, 5.0), (20, np.inf)])
@pytest.mark.parametrize("n,kind,qkind", [(300, "nan_axis", "plain"), (5000, "nan_axis", "plain"),
                                          (6000, "nan_most", "odd"), (5000, "piles", "plain"),
                                          (25, "box", "odd"), (5000, "box", "odd"), (90, "infinite", "odd"),
                                          (4000, "infinite", "odd")])
def test_odd_sets(n, kind, qkind, k, radius, noalloc):
    rs = np.random.RandomState(n + k)
    p = records(kind, n, rs)
    q = queries(qkind, p, rs)
    bi, bd = brute(p, q, k, radius)
    qd = torch.from_numpy(q).cuda()
    idx = torch.zeros((len(q), k), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((len(q), k), dtype=torch.float32, device="cuda")
    if noalloc:
        pd = torch.from_numpy(p).cuda()
        s = photonmap.load().pm_knn_noalloc(pd.data_ptr(), n, qd.data_ptr(), len(q), k, float(radius),
                                            idx.data_ptr(), d2.data_ptr(), None)
        torch.cuda.synchronize()
        assert s == 0
    else:
        sc, cf = photonmap.preset(1)
        with photonmap.Context(0) as ctx:
            ctx.set_scene(sc, cf)
            for m in (0, 1):
                ctx.set_photons(m, p, np.ones_like(p))
            ctx.build()
            ctx.knn(1, qd.data_ptr(), len(q), k, float(radius), idx.data_ptr(), d2.data_ptr())
            torch.cuda.synchronize()
    np.testing.assert_array_equal(idx.cpu().numpy().view(np.uint32), bi)
    np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), bd.view(np.uint32))
