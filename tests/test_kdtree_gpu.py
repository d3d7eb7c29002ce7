"""The kd-tree build through pm_set_photons + pm_build + pm_knn: the k
nearest records of any point set are those of a brute-force sort by
(squared distance, index), whatever the set's size and shape.

Sizes sit at the edges of the build's parts: leaves of 32, warp splits of 64
and 128, subtrees of 2,048 records, tiles of 4,096, clusters of 32,768, one to
seven split levels, both maps in shared launches and (above 4M records) apart."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402

pytestmark = pytest.mark.gpu


def shaped(kind, n, rs):
    p = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5], size=(n, 3)).astype(np.float32)
    if kind == "wall":        # most records share one coordinate
        p[: n - n // 7, 1] = 0.0
    elif kind == "point":     # most records are one point
        p[: n - n // 5] = np.float32([0.1, 0.2, 0.3])
    elif kind == "outlier":   # a tight cluster and one record far away
        p[:] = np.float32([0.3, 0.3, 0.3]) + (p - np.float32([0, 0.5, 0])) * np.float32(1e-4)
        p[n // 2] = (50.0, -40.0, 30.0)
    elif kind == "nonfinite":
        p[:: 17] = np.inf
        p[1:: 23] = np.nan
        p[2:: 29, 0] = -np.inf
    return p


def brute(p, q, k, radius):
    """(index, squared distance) lists in the search's own arithmetic."""
    r2 = np.float32(radius) * np.float32(radius)
    idx = np.full((len(q), k), 0xFFFFFFFF, np.uint32)
    d2 = np.full((len(q), k), r2, np.float32)
    with np.errstate(invalid="ignore", over="ignore"):
        for i, x in enumerate(q):
            d = p - x
            s = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
            c = np.flatnonzero(s <= r2)
            c = c[np.lexsort((c, s[c]))][:k]
            idx[i, : len(c)] = c
            d2[i, : len(c)] = s[c]
    return idx, d2


CASES = [(n, "box", ls) for n in (1, 32, 33, 64, 65, 128, 129, 2047, 2048, 2049, 4096, 4097, 8193,
                                              32767, 32769, 65537)
         for ls in (32,)]
CASES += [(n, "box", ls) for n in (100, 128, 129, 5000, 131073) for ls in (64, 128)]
CASES += [(n, kind, 32) for n in (3000, 40001, 300007) for kind in ("wall", "point", "outlier", "nonfinite")]


@pytest.mark.parametrize("n,kind,leaf", CASES)
def test_knn_over_any_point_set(n, kind, leaf):
    rs = np.random.RandomState(n + leaf)
    sc, cf = photonmap.preset(1)
    cf.surface_photons, cf.volume_photons, cf.leaf_size = n, 777, leaf
    maps = [shaped(kind, n, rs), shaped("box", 777, rs)]
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        for m in (0, 1):
            pos = np.zeros((len(maps[m]), 4), np.float32)
            pos[:, :3] = maps[m]
            ctx.set_photons(m, pos, np.ones_like(pos))
        ctx.build()
        for m, k, radius in ((0, 100, 0.2), (0, 9, 3.0), (1, 32, 0.3)):
            p = maps[m]
            q = np.zeros((60, 4), np.float32)
            q[:, :3] = rs.uniform(-0.6, 1.1, size=(60, 3))
            near = p[rs.randint(0, len(p), 30)]
            q[:30, :3] = np.where(np.isfinite(near), near, 0.0) + rs.normal(0, 1e-5, (30, 3)).astype(np.float32)
            qd = torch.from_numpy(q).cuda()
            idx = torch.zeros((60, k), dtype=torch.int32, device="cuda")
            d2 = torch.zeros((60, k), dtype=torch.float32, device="cuda")
            ctx.knn(m, qd.data_ptr(), 60, k, radius, idx.data_ptr(), d2.data_ptr())
            torch.cuda.synchronize()
            bi, bd = brute(p, q[:, :3], k, radius)
            np.testing.assert_array_equal(idx.cpu().numpy().view(np.uint32), bi)
            np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), bd.view(np.uint32))


def test_large_map_apart_from_the_other():
    """Above 4M records in all the maps are built one after the other."""
    n = (1 << 22) + 4097
    rs = np.random.RandomState(1)
    sc, cf = photonmap.preset(1)
    cf.surface_photons, cf.volume_photons = n, 5000
    maps = [shaped("wall", n, rs), shaped("box", 5000, rs)]
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        for m in (0, 1):
            pos = np.zeros((len(maps[m]), 4), np.float32)
            pos[:, :3] = maps[m]
            ctx.set_photons(m, pos, np.ones_like(pos))
        ctx.build()
        q = np.zeros((8, 4), np.float32)
        q[:, :3] = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5], size=(8, 3))
        q[:4, 1] = 0.0
        for m in (0, 1):
            qd = torch.from_numpy(q).cuda()
            idx = torch.zeros((8, 64), dtype=torch.int32, device="cuda")
            d2 = torch.zeros((8, 64), dtype=torch.float32, device="cuda")
            ctx.knn(m, qd.data_ptr(), 8, 64, 0.3, idx.data_ptr(), d2.data_ptr())
            torch.cuda.synchronize()
            bi, bd = brute(maps[m], q[:, :3], 64, 0.3)
            np.testing.assert_array_equal(idx.cpu().numpy().view(np.uint32), bi)
            np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), bd.view(np.uint32))
