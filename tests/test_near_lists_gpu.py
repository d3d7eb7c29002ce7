"""The tracer's sphere lists (scenes of many spheres with large maps) against
the FP32 oracle, which tests every sphere: every record bit for bit. Spheres
that overlap, stick out of the box, are tiny or fill it; lights inside, on
the box and outside it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu

TARGET = 500000  # enough for the lists at 48 spheres and more


@pytest.mark.parametrize("spheres,radii,light", [
    (64, (0.05, 0.3), (0.0, 0.95, 0.0)),
    (64, (0.002, 0.02), (0.5, 0.5, -0.5)),
    (48, (0.02, 0.1), (0.0, 1.4, 0.0)),
    (57, (0.2, 0.6), (-0.1, 0.4, 0.2)),
    (64, (0.01, 0.4), (0.0, 0.5, -1.5)),
])
def test_emission_through_the_lists(spheres, radii, light):
    rs = np.random.RandomState(spheres)
    sc, cf = photonmap.preset(3, 0x5EED0007)
    sc.num_spheres = spheres
    for i in range(spheres):
        sc.spheres[i][0], sc.spheres[i][1], sc.spheres[i][2] = rs.uniform([-0.6, -0.1, -0.6], [0.6, 1.1, 0.6])
        sc.spheres[i][3] = rs.uniform(*radii)
    for a in range(3):
        sc.light[a] = light[a]
    cf.surface_photons, cf.volume_photons, cf.max_paths = TARGET, 2000, 60000
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        ctx.emit()
        het = oracle.noise_grid(sc, cf)
        m = oracle.emit(sc, cf, het)
        assert m.sizes[0] > 1000
        for mid, (op, ow) in enumerate([(m.spos, m.spow), (m.vpos, m.vpow)]):
            pos, pw = ctx.photons_soa(mid)
            assert len(pos) == len(op)
            np.testing.assert_array_equal(pos.view(np.uint32), op.view(np.uint32))
            np.testing.assert_array_equal(pw.view(np.uint32), ow.view(np.uint32))
