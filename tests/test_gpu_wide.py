"""GPU parity of the four-wide traversal where its records and its ray rules
can go wrong: trees of a few triangles up to the edges of the emit's blocks,
and rays whose slab tests meet 0 * inf (parallel to an axis, on a box face).
Every hit record and shadow mask equals the oracle's bit for bit."""
import numpy as np
import pytest

from rtgb import abi, capi, scenes

pytestmark = pytest.mark.gpu


def _samples(o, d):
    s = np.zeros(o.shape[0], abi.SAMPLE_DTYPE)
    s["ori"][:, :3] = o
    s["dir"][:, :3] = d
    with np.errstate(divide="ignore"):
        s["inv_dir"][:, :3] = np.float32(1) / d.astype(np.float32)
    s["tmin"], s["tmax"] = 0.0001, 1e37
    s["contribution"] = 1.0
    return s


def _compare(ctx, orc, sc, smp, min_leaf=1):
    g, o = capi.Scene(ctx, sc), orc.new_scene(sc)
    g.build(30, min_leaf)
    o.build(30, min_leaf, 0)
    n = smp.shape[0]
    smp_d, hit_d = ctx.to_device(smp), ctx.alloc(64 * n)
    hit_d.zero()
    g.trace(smp_d, n, hit_d)
    g.shadow(smp_d, n, hit_d)
    ctx.sync()
    got, ref = hit_d.read(abi.HIT_DTYPE), o.trace(smp)
    o.shadow(smp, ref)
    m = ref["hit"] == 1
    assert np.array_equal(got["hit"], ref["hit"])
    for f in ("id", "t", "inverse_n", "shadow_hit"):
        assert np.array_equal(got[f][m], ref[f][m]), f
    for f in ("n", "hit_point"):
        assert np.array_equal(got[f][m][:, :3], ref[f][m][:, :3]), f
    assert ctx.device_status() == 0
    return int(m.sum())


def _random_rays(n, seed):
    r = np.random.default_rng(seed)
    o = r.uniform(-3, 3, (n, 3)).astype(np.float32)
    d = (r.uniform(-1, 1, (n, 3)) - o).astype(np.float32)
    d /= np.linalg.norm(d, axis=1, keepdims=True).astype(np.float32)
    return _samples(o, d)


@pytest.mark.parametrize("n,min_leaf", [(1, 1), (3, 1), (4, 1), (5, 1), (6, 4), (7, 1), (9, 1), (16, 4),
                                        (33, 1), (257, 1), (511, 256), (512, 1), (513, 1), (4097, 2),
                                        (4609, 1), (40000, 1)])
def test_trees_of_every_size(ctx, orc, n, min_leaf):
    sc = scenes.soup(n, seed=n, offset_sigma=max(0.03, 0.5 / n ** 0.4))
    assert _compare(ctx, orc, sc, _random_rays(4096, n), min_leaf) > 0


def _grid_scene(light_dir):
    """A height field on whole numbers: boxes of zero thickness that share faces."""
    ter = scenes.Terrain(24, 24, extent=(0.0, 24.0, 0.0, 24.0), n_spheres=3, seed=4)
    pos, nrm = ter.frame_vertices(0)
    g = ter.n_grid_verts
    pos[:g, 1] = np.round(pos[:g, 1])
    lights = abi.make_lights((0.1,) * 3, [dict(type=abi.RT_DIR_L, dir=light_dir),
                                          dict(type=abi.RT_POINT_L, pos=(12.0, 9.0, 12.0))])
    return scenes.Scene(pos, nrm, ter.idx, ter.mats, ter.mat_map, lights)


@pytest.mark.parametrize("light_dir", [(0.0, -1.0, 0.0), (-1.0, -0.0, 0.0), (0.0, -0.6, 0.8)])
def test_axis_parallel_rays(ctx, orc, light_dir):
    """Origins on whole numbers (on box faces), directions with one or two
    zero components of either sign, a share of ordinary rays among them."""
    r = np.random.default_rng(8)
    n = 8192
    o = r.integers(-1, 26, (n, 3)).astype(np.float32)
    o[:, 1] = r.integers(-4, 6, n)
    d = r.choice(np.array([-1.0, -0.0, 0.0, 1.0, 0.5], np.float32), (n, 3))
    d[(d == 0).all(axis=1)] = (0.0, -1.0, 0.0)
    d[::7] = r.normal(size=d[::7].shape)
    assert _compare(ctx, orc, _grid_scene(light_dir), _samples(o, d)) > 500
