"""pm_knn's choice between the list search (one launch, maps with few records
in a query's reach) and the selection (two) goes by the box of the records,
not of the scene. Either way the results are a brute-force sort's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402
from test_kdtree_gpu import brute  # noqa: E402

pytestmark = pytest.mark.gpu

UNIT = ([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5])
# points, box, radius, launches: about 10, 400, 10,000, 0.4, 8 and 5,600 expected in reach
CASES = [(20000, UNIT, 0.05, 1), (20000, UNIT, 0.17, 2), (20000, ([0.1, 0.1, 0.1], [0.2, 0.2, 0.2]), 0.05, 2),
         (100000, ([-5.0, 0.0, -5.0], [5.0, 10.0, 5.0]), 0.1, 1), (1000, ([9.0, 9.0, 3.0], [10.0, 10.0, 3.0]), 0.05, 1),
         (20000, ([9.0, 9.0, 3.0], [10.0, 10.0, 3.0]), 0.3, 2)]


@pytest.mark.parametrize("n,box,radius,launches", CASES)
def test_route_by_the_records_own_box(n, box, radius, launches):
    rs = np.random.RandomState(n)
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = rs.uniform(box[0], box[1], size=(n, 3))
    q = np.zeros((50, 4), np.float32)
    q[:, :3] = rs.uniform(box[0], box[1], size=(50, 3))
    sc, cf = photonmap.preset(1)
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        for m in (0, 1):
            ctx.set_photons(m, p, np.ones_like(p))
        ctx.build()
        qd = torch.from_numpy(q).cuda()
        for k in (1, 40):
            idx = torch.zeros((50, k), dtype=torch.int32, device="cuda")
            d2 = torch.zeros((50, k), dtype=torch.float32, device="cuda")
            before = photonmap.load().pm_kernel_launches()
            ctx.knn(1, qd.data_ptr(), 50, k, radius, idx.data_ptr(), d2.data_ptr())
            assert photonmap.load().pm_kernel_launches() - before == launches
            torch.cuda.synchronize()
            bi, bd = brute(p[:, :3], q[:, :3], k, radius)
            np.testing.assert_array_equal(idx.cpu().numpy().view(np.uint32), bi)
            np.testing.assert_array_equal(d2.cpu().numpy().view(np.uint32), bd.view(np.uint32))


def test_left_queries_cost_a_list_search():
    """20,000 queries at a pile of 100,000 records, which no warp's registers
    hold, so that all are left to the list search: at most 2.5 times the list
    search's own route (a few records far off make the map thin), which does the
    same work. Left queries that one warp in 32 serves took 8 times as long."""
    n, nq, k = 100000, 20000, 32
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = np.float32([0.1, 0.5, 0.1])
    far = p.copy()
    far[:98 * 8: 98, :3] = [[a, b, c] for a in (-100.0, 100.0) for b in (-100.0, 100.0) for c in (-100.0, 100.0)]
    qd = torch.from_numpy(p[:nq].copy()).cuda()
    idx = torch.zeros((nq, k), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((nq, k), dtype=torch.float32, device="cuda")
    sc, cf = photonmap.preset(1)
    times, launches = [], []
    for records in (far, p):
        with photonmap.Context(0) as ctx:
            ctx.set_scene(sc, cf)
            for m in (0, 1):
                ctx.set_photons(m, records, np.ones_like(records))
            ctx.build()
            stream = torch.cuda.current_stream().cuda_stream
            best = 1e9
            for _ in range(5):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                before = photonmap.load().pm_kernel_launches()
                a.record()
                ctx.knn(1, qd.data_ptr(), nq, k, 0.05, idx.data_ptr(), d2.data_ptr(), stream)
                b.record()
                torch.cuda.synchronize()
                best = min(best, a.elapsed_time(b))
            launches.append(photonmap.load().pm_kernel_launches() - before)
            times.append(best)
        assert (d2 == 0).all()
    print("list search %.2f ms, left to it %.2f ms" % tuple(times))
    assert launches == [1, 2]
    assert times[1] < 2.5 * times[0], times
