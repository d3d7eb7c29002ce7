"""pm_knn_noalloc's results at the sizes where its build changes: one subtree
(no root box) to 2,048 points, clusters alone to 32,768, split levels beyond;
each after a larger call on the same scratch, and with points that are not
finite, which the root's box leaves out."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402
from test_kdtree_gpu import brute, shaped  # noqa: E402

pytestmark = pytest.mark.gpu


def noalloc(p, q, k, radius):
    pd = np.zeros((len(p), 4), np.float32)
    pd[:, :3] = p
    pd, qd = torch.from_numpy(pd).cuda(), torch.from_numpy(q).cuda()
    idx = torch.zeros((len(q), k), dtype=torch.int32, device="cuda")
    d2 = torch.zeros((len(q), k), dtype=torch.float32, device="cuda")
    s = photonmap.load().pm_knn_noalloc(pd.data_ptr(), len(p), qd.data_ptr(), len(q), k, radius, idx.data_ptr(),
                                        d2.data_ptr(), None)
    torch.cuda.synchronize()
    assert s == 0, s
    return idx.cpu().numpy().view(np.uint32), d2.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("kind", ["box", "nonfinite", "point"])
@pytest.mark.parametrize("n", [1, 33, 2048, 2049, 4097, 20011, 32768, 32769, 131072])
def test_results_at_every_form_of_the_build(n, kind):
    rs = np.random.RandomState(n)
    sets = [shaped("wall", min(2 * n + 5000, 131072), rs), shaped(kind, n, rs)]
    for p in sets:
        q = np.zeros((40, 4), np.float32)
        q[:, :3] = rs.uniform([-0.6, -0.1, -0.6], [0.6, 1.1, 0.6], size=(40, 3))
        near = p[rs.randint(0, len(p), 20)]
        q[:20, :3] = np.where(np.isfinite(near), near, 0.0)
        for k, radius in ((7, 0.2), (100, 0.5)):
            gi, gd = noalloc(p, q, k, radius)
            bi, bd = brute(p, q[:, :3], k, radius)
            np.testing.assert_array_equal(gi, bi)
            np.testing.assert_array_equal(gd, bd.view(np.uint32))
