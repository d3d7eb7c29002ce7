"""pm_radius_gather far beyond a scene's range: distances of 10^9 and
exposures at which the weight of a record is large, and its factors together
beyond a float, against the FP64 oracle. Records that face away add zero. Each
sum has 40 terms of a few float roundings, added with compensation: 2e-6
relative, and the same of the largest for sums that are nearly zero."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far,exposure", [(1e9, 2e-30), (1e9, -2e-30), (1e6, 1e-32), (1e9, 1e20), (1.0, 2e-30)])
def test_weights_beyond_a_float_in_their_factors(far, exposure):
    rs = np.random.RandomState(7)
    n, nq = 40, 33
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5], size=(n, 3))
    pw = np.zeros((n, 4), np.float32)
    pw[:, :3] = rs.uniform(0.1, 1.0, size=(n, 3))
    pw[:, 3] = rs.randint(-2 ** 31, 2 ** 31 - 1, n).astype(np.int32).view(np.float32)
    pw[~np.isfinite(pw[:, 3]), 3] = 0.0
    pts, nrm = np.zeros((nq, 4), np.float32), np.zeros((nq, 4), np.float32)
    v = rs.standard_normal((nq, 3)).astype(np.float32)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    pts[:, :3] = v * np.float32(far)
    nrm[:, :3] = rs.standard_normal((nq, 3)).astype(np.float32) * np.float32(1e-3)
    sq_radius = float(np.float32(4.0 * far * far))
    sc, cf = photonmap.preset(1)
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        for m in (0, 1):
            ctx.set_photons(m, pos, pw)
        ctx.build()
        got_pos, got_pw = ctx.photons_soa(0)
        pd, nd = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()
        out = torch.zeros((nq, 4), dtype=torch.float32, device="cuda")
        ctx.radius_gather(0, pd.data_ptr(), nd.data_ptr(), nq, sq_radius, exposure, out.data_ptr())
        torch.cuda.synchronize()
    got = out.cpu().numpy()[:, :3].astype(np.float64)
    ref = oracle.radius_gather(got_pos, got_pw, pts, nrm, sq_radius, exposure)
    scale = np.abs(ref).max()
    assert 0 < scale < 3e38
    np.testing.assert_allclose(got, ref, rtol=2e-6, atol=2e-6 * scale)


@pytest.mark.parametrize("scale", [1e-36, 1e-25, 1e-16, 1e-3, 1e6])
def test_normals_of_any_length(scale):
    """A weight is proportional to the normal's length; that of a tiny one is
    within a float's spacing, which the margins cover ten times."""
    rs = np.random.RandomState(9)
    n, nq = 400, 33
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5], size=(n, 3))
    pw = np.zeros((n, 4), np.float32)
    pw[:, :3] = rs.uniform(0.1, 1.0, size=(n, 3))
    pw[:, 3] = rs.randint(-2 ** 31, 2 ** 31 - 1, n).astype(np.int32).view(np.float32)
    pw[~np.isfinite(pw[:, 3]), 3] = 0.0
    pts, nrm = np.zeros((nq, 4), np.float32), np.zeros((nq, 4), np.float32)
    pts[:, :3] = pos[:nq, :3] + np.float32(0.01)
    nrm[:, :3] = rs.standard_normal((nq, 3)).astype(np.float32) * np.float32(scale)
    sc, cf = photonmap.preset(1)
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        for m in (0, 1):
            ctx.set_photons(m, pos, pw)
        ctx.build()
        got_pos, got_pw = ctx.photons_soa(0)
        pd, nd = torch.from_numpy(pts).cuda(), torch.from_numpy(nrm).cuda()
        out = torch.zeros((nq, 4), dtype=torch.float32, device="cuda")
        ctx.radius_gather(0, pd.data_ptr(), nd.data_ptr(), nq, 0.1, 0.5, out.data_ptr())
        torch.cuda.synchronize()
    got = out.cpu().numpy()[:, :3].astype(np.float64)
    ref = oracle.radius_gather(got_pos, got_pw, pts, nrm, 0.1, 0.5)
    top = np.abs(ref).max()
    assert top > 0
    np.testing.assert_allclose(got, ref, rtol=2e-6, atol=2e-6 * top)
