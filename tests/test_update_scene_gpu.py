"""pm_update_scene with the tracer's sphere lists: it allocates nothing when
the sphere count changes across the sizes of the lists, and the records that
follow are those of a context that was given the scene at first."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402

pytestmark = pytest.mark.gpu


def scene(spheres, seed=1):
    rs = np.random.RandomState(seed)
    sc, cf = photonmap.preset(3, 0x5EED0007)
    sc.num_spheres = spheres
    for i in range(spheres):
        sc.spheres[i][0], sc.spheres[i][1], sc.spheres[i][2] = rs.uniform([-0.5, 0.0, -0.5], [0.5, 1.0, 0.5])
        sc.spheres[i][3] = rs.uniform(0.03, 0.2)
    cf.surface_photons, cf.volume_photons, cf.max_paths = 1000000, 2000, 60000
    return sc, cf


def records(ctx):
    return [a.view(np.uint32) for m in (0, 1) for a in ctx.photons_soa(m)]


def fresh(sc, cf):
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        ctx.emit()
        return records(ctx)


def test_sphere_counts_change_without_allocation():
    torch.cuda.set_device(0)
    first, cf = scene(5)
    fresh(*scene(64))  # every kernel loaded
    with photonmap.Context(0) as ctx:
        ctx.set_scene(first, cf)
        ctx.emit()
        free, _ = torch.cuda.mem_get_info()
        for n in (64, 30, 0, 45):
            sc, _ = scene(n, n)
            ctx.update_scene(sc)
            assert torch.cuda.mem_get_info()[0] == free, n
            ctx.emit()
            assert torch.cuda.mem_get_info()[0] == free, n
            for got, want in zip(records(ctx), fresh(sc, cf)):
                np.testing.assert_array_equal(got, want)


def launches(ctx):
    n = photonmap.load().pm_kernel_launches()
    ctx.emit()
    return photonmap.load().pm_kernel_launches() - n


def test_lists_are_kept_while_spheres_and_box_are():
    """One launch builds the lists: an emission after a camera, light, medium or
    material change has as many launches as a repeated one, and one more after
    a sphere, the box or the count has changed. The records are always those
    of a fresh context."""
    sc, cf = scene(64)

    def changed(what):
        if what == "camera":
            sc.cam_pos[0] += 0.1
        elif what == "light":
            sc.light[0], sc.light_power = 0.1, sc.light_power * 2
        elif what == "medium":
            sc.sigma_a, sc.hg_g = 0.3, 0.1
        elif what == "material":
            sc.sphere_mat[3].kind = photonmap.MAT_MIRROR
        elif what == "sphere":
            sc.spheres[5][1] += 0.05
        elif what == "radius":
            sc.spheres[63][3] *= 0.5
        elif what == "box":
            sc.box_max[1] += 0.25
        elif what == "count":
            sc.num_spheres = 63

    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        assert launches(ctx) == launches(ctx) + 1
        kept = launches(ctx)
        for what, built in [("camera", 0), ("light", 0), ("medium", 0), ("material", 0), ("sphere", 1), ("camera", 0),
                            ("radius", 1), ("box", 1), ("count", 1)]:
            changed(what)
            ctx.update_scene(sc)
            assert launches(ctx) == kept + built, what
            for got, want in zip(records(ctx), fresh(sc, cf)):
                np.testing.assert_array_equal(got, want)
            assert launches(ctx) == kept, what
