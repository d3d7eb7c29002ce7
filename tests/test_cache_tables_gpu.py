"""The cache at table sizes on both sides of each kind of level: 2^12 to 2^22
entries have 0 to 8 dense levels at the default resolutions, and inference is
compiled for each number of them. The encoding, forward and backward pass and
the cached values against the FP64 oracle; grids of other level counts and
resolutions take the general form.

Tolerances: features are sums of 8 products of fp32 weights and fp16 table
values below 0.5 (2e-5), the network's inputs, weights and activations are
bf16 (2^-9 each through 5 layers: 1e-2 of the norm, 2e-2 for gradients)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
import photonmap  # noqa: E402
import cache_oracle as co  # noqa: E402

pytestmark = pytest.mark.gpu

TABLES = [(12, 0, {}), (13, 1, {}), (14, 2, {}), (15, 3, {}), (17, 4, {}), (19, 5, {}), (20, 6, {}),
          (15, 16, dict(base_res=4, max_res=30)), (15, 2, dict(levels=12)), (15, 2, dict(base_res=20, max_res=4000))]


def dense_levels(res, log2_table):
    return sum((int(r) + 1) ** 3 <= 1 << log2_table for r in res)


@pytest.fixture(scope="module")
def ctx():
    with photonmap.Context(0) as c:
        sc, cf = photonmap.preset(2, 0x5EED0001)
        cf.surface_photons = cf.volume_photons = 20000
        cf.width = cf.height = 40
        c.set_scene(sc, cf)
        c.emit()
        c.build()
        c.sc = sc
        yield c


def geometry(sc):
    return (np.array([list(sc.spheres[i]) for i in range(sc.num_spheres)], np.float64),
            [int(sc.planes[i][0]) for i in range(sc.num_planes)])


def norm_error(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("log2_table,dense,grid", TABLES)
def test_encoding_and_gradients(ctx, log2_table, dense, grid):
    cfg = ctx.cache_enable(log2_table=log2_table, **grid)
    w, t, res = ctx.cache_params()
    assert dense_levels(res, log2_table) == dense
    rng = np.random.default_rng(log2_table)
    t = rng.uniform(-0.3, 0.3, t.shape).astype(np.float32)
    ctx.cache_set_params(table=t)
    qa, qd = ctx.cache_queries()
    pick = rng.choice(len(qa), 700, replace=len(qa) < 700)
    qa, qd = qa[pick], qd[pick]
    target = np.zeros((700, 4), np.float32)
    target[:, :3] = rng.uniform(0.0, 2.0, (700, 3))
    out = ctx.cache_debug_step(qa, qd, target, target_scale=1.7)
    assert ctx.cache_stats().tc_status == 0
    lo, inv = co.grid_box(ctx.sc.box_min, ctx.sc.box_max)
    x = co.features(qa, qd, lo, inv, t, res, log2_table, *geometry(ctx.sc))
    np.testing.assert_allclose(out["x"][:, :32], x[:, :32], rtol=0, atol=2e-5)
    ref = co.mlp_step(x, w, target[:, :3] / np.float32(1.7), eps=cfg.loss_eps)
    assert norm_error(out["y"][:, :3], ref["y"]) < 1e-2
    assert norm_error(out["w_grad"], ref["w_grad"]) < 2e-2
    tg = co.table_grad(co.unit_pos(qa[:, :3], lo, inv), ref["dx"], res, log2_table)
    for l in range(len(res)):  # each level: gradients at the entries that were read
        assert norm_error(out["table_grad"][l], tg[l]) < 2e-2, l


@pytest.mark.parametrize("log2_table,dense,grid", TABLES + [(21, 7, {}), (22, 8, {})])
def test_cached_values(ctx, log2_table, dense, grid):
    ctx.cache_enable(log2_table=log2_table, train_samples=1 << 13, batch=1 << 12, **grid)
    rng = np.random.default_rng(log2_table)
    w, t, res = ctx.cache_params()
    assert dense_levels(res, log2_table) == dense
    ctx.cache_train(2)  # fixes the target scale
    ctx.cache_set_params(table=rng.uniform(-0.3, 0.3, t.shape).astype(np.float32))
    w, t, res = ctx.cache_params()
    ctx.render_cached(torch.zeros((1600, 4), device="cuda").data_ptr(), None, 0)
    torch.cuda.synchronize()
    qa, qd = ctx.cache_queries()
    pick = rng.choice(len(qa), 3000, replace=False)
    got = ctx.cache_values()[pick, :3]
    lo, inv = co.grid_box(ctx.sc.box_min, ctx.sc.box_max)
    x = co.features(qa[pick], qd[pick], lo, inv, t, res, log2_table, *geometry(ctx.sc))
    y = co.mlp_step(x, w, np.zeros((3000, 3)))["y"]
    ref = np.maximum(y, 0.0) * np.float32(ctx.cache_stats().target_scale)
    assert ctx.cache_stats().tc_status == 0
    assert (ref > 0).mean() > 0.1
    assert norm_error(got, ref) < 1e-2
