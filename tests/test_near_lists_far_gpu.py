"""The tracer's sphere lists in boxes far from the origin, where a float's
spacing is coarse against a cell, and in boxes without a finite size: every
record is the FP32 oracle's, which tests every sphere, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402
import oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift,size,infinite", [(500.0, 1.0, False), (2000.0, 1.0, False), (2e4, 1.0, False),
                                                 (1e5, 1.0, False), (1e6, 1.0, False), (4e6, 1.0, False), (0.0, 1.0, True), (0.0, 1e18, False),
                                                 (0.0, 0.02, False)])
def test_emission_far_from_the_origin(shift, size, infinite):
    rs = np.random.RandomState(5)
    sc, cf = photonmap.preset(3, 0x5EED0007)
    at = np.float64([shift, -shift, shift])
    for i in range(64):
        c = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5]) * size + at
        sc.spheres[i][0], sc.spheres[i][1], sc.spheres[i][2] = c
        sc.spheres[i][3] = rs.uniform(0.03, 0.25) * size
    for a in range(3):
        sc.box_min[a] = sc.box_min[a] * size + at[a]
        sc.box_max[a] = sc.box_max[a] * size + at[a]
        sc.light[a] = sc.light[a] * size + at[a]
    for i in range(sc.num_planes):
        sc.planes[i][1] = sc.planes[i][1] * size + at[int(sc.planes[i][0])]
    if infinite:
        sc.box_max[1] = np.inf
    sc.het_res, sc.sigma_s, sc.sigma_a = 0, 0.0, 0.0
    cf.surface_photons, cf.volume_photons, cf.max_paths = 500000, 2000, 40000
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        ctx.emit()
        m = oracle.emit(sc, cf, oracle.noise_grid(sc, cf))
        assert m.sizes[0] > 1000
        for mid, (op, ow) in enumerate([(m.spos, m.spow), (m.vpos, m.vpow)]):
            pos, pw = ctx.photons_soa(mid)
            assert len(pos) == len(op)
            np.testing.assert_array_equal(pos.view(np.uint32), op.view(np.uint32))
            np.testing.assert_array_equal(pw.view(np.uint32), ow.view(np.uint32))
