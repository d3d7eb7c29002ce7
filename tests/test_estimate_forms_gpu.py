"""The estimate pass's forms, on both sides of the query counts that choose
them (152 SMs): groups of 8 below 272,384 queries, then groups of 32, one, two
(from 2.2M) or four (from 34.9M) to a warp's chunk. Every image is the
single-kernel render's, which has one list search a query, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402

pytestmark = pytest.mark.gpu

WARPS = 152 * 28
EDGES = [0, 64 * WARPS, 64 * 8 * WARPS, 128 * 64 * WARPS, 1 << 40]  # form f: EDGES[f] <= queries < EDGES[f + 1]


def images(ctx, cf, render):
    rad = torch.zeros((cf.width * cf.height, 4), dtype=torch.float32, device="cuda")
    rgba = torch.zeros((cf.width * cf.height, 4), dtype=torch.uint8, device="cuda")
    render(rad.data_ptr(), rgba.data_ptr())
    torch.cuda.synchronize()
    return rad.cpu().numpy().view(np.uint32), rgba.cpu().numpy()


@pytest.mark.parametrize("form,size,step,k", [(0, (79, 61), 0.02, 64), (0, (109, 107), 0.02, 33), (1, (121, 115), 0.02, 64),
                                              (1, (315, 313), 0.02, 100), (2, (330, 325), 0.02, 9), (2, (901, 899), 0.01, 32),
                                              (3, (930, 925), 0.01, 64)])
def test_image_is_the_single_kernels(form, size, step, k):
    sc, cf = photonmap.preset(1, 0x5EED0003)
    cf.surface_photons = cf.volume_photons = 60000
    cf.width, cf.height = size
    cf.march_step, cf.k = step, k
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        ctx.emit()
        ctx.build()
        got = images(ctx, cf, ctx.render)
        st = ctx.stats()
        queries = st.surface_gathers + st.volume_gathers
        print("%d queries" % queries)
        assert EDGES[form] <= queries < EDGES[form + 1], queries
        want = images(ctx, cf, ctx.render_single_kernel)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("form,size", [(1, 64), (2, 400), (3, 1500)])
def test_batch_of_large_frames(form, size):
    """The pass over many scenes (never groups of 8): two scenes' frames, each
    the single scene's."""
    scenes, cfgs = [], []
    for i in (0, 3):
        sc, cf = photonmap.batch_scene(i, 0x5EED0005)
        cf.surface_photons = cf.volume_photons = 30000
        cf.width = cf.height = size
        cf.march_step, cf.k, cf.max_paths = 0.04, 33, 240000
        scenes.append(sc)
        cfgs.append(cf)
    with photonmap.Context(0) as ctx:
        b = photonmap.Batch(ctx, scenes, cfgs)
        for i in range(2):
            b.set_tune(i, query_list=1)
        b.frame()
        torch.cuda.synchronize()
        got = [b.read(i)[0].view(np.uint32) for i in range(2)]
        queries = sum(b.stats(i).surface_gathers + b.stats(i).volume_gathers for i in range(2))
        print("%d queries" % queries)
        assert queries >= EDGES[2 if form == 2 else 3 if form == 3 else 0], queries
        b.close()
        for i, (sc, cf) in enumerate(zip(scenes, cfgs)):
            ctx.set_scene(sc, cf)
            ctx.emit()
            ctx.build()
            want = images(ctx, cf, ctx.render_single_kernel)[0]
            np.testing.assert_array_equal(got[i], want, err_msg="scene %d" % i)


@pytest.mark.parametrize("photons,k", [(40, 100), (300, 100), (5000, 20)])
def test_infinite_radius(photons, k):
    """Nothing bounds a set but the map itself, which may hold fewer than k."""
    sc, cf = photonmap.preset(1, 0x5EED0003)
    cf.surface_photons = cf.volume_photons = photons
    cf.width, cf.height = 40, 33
    cf.march_step, cf.k, cf.radius = 0.05, k, float("inf")
    with photonmap.Context(0) as ctx:
        ctx.set_scene(sc, cf)
        ctx.emit()
        ctx.build()
        got, want = images(ctx, cf, ctx.render), images(ctx, cf, ctx.render_single_kernel)
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
