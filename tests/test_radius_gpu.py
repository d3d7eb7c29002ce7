"""pm_radius_gather's weight in single-precision pairs and, for exposures
whose reciprocal they cannot hold, in double precision, against the FP64
oracle. A query sums n non-negative terms, each within a few float roundings
of its value, by compensated sums: 1e-6 relative covers the terms, and the
records whose distance rounds across the radius (the weight is not zero
there) need an absolute margin of one term."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exposure", [50.0, 1.0, -2.0, 3e-7, 1e15, 5e25, 1e-32])
def test_weight_over_the_range_of_exposures(exposure):
    rs = np.random.RandomState(3)
    n, nq = 5000, 257
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5], size=(n, 3))
    pw = np.zeros((n, 4), np.float32)
    pw[:, :3] = rs.uniform(0.1, 1.0, size=(n, 3))
    pw[:, 3] = rs.randint(-2 ** 31, 2 ** 31 - 1, n).astype(np.int32).view(np.float32)
    pw[~np.isfinite(pw[:, 3]), 3] = 0.0
    pts, nrm = np.zeros((nq, 4), np.float32), np.zeros((nq, 4), np.float32)
    pts[:, :3] = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5], size=(nq, 3))
    v = rs.standard_normal((nq, 3)).astype(np.float32)
    nrm[:, :3] = v / np.linalg.norm(v, axis=1, keepdims=True)
    sc, cf = photonmap.preset(1)
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        ctx.set_photons(0, pos, pw)
        ctx.set_photons(1, pos[:10], pw[:10])
        ctx.build()
        got_pos, got_pw = ctx.photons_soa(0)
        pd, nd = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()
        out = torch.zeros((nq, 4), dtype=torch.float32, device="cuda")
        ctx.radius_gather(0, pd.data_ptr(), nd.data_ptr(), nq, 0.01, exposure, out.data_ptr())
        torch.cuda.synchronize()
    got = out.cpu().numpy()[:, :3].astype(np.float64)
    ref = oracle.radius_gather(got_pos, got_pw, pts, nrm, 0.01, exposure)
    scale = np.abs(ref).max()
    assert scale > 0 and np.isfinite(scale)
    np.testing.assert_allclose(got, ref, rtol=2e-6, atol=1e-6 * scale)
