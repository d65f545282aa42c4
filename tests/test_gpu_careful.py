"""Rays whose slab tests meet 0 * inf or boxes at infinity: parallel to an axis,
in the plane of a flat box, without an upper bound, from infinite or NaN
origins.  Each set runs on both sides of the line between four lanes and one
lane per ray, mixed with ordinary rays, and every hit record and shadow mask
equals the oracle's bit for bit.  Parallel rays cost no more than tilted ones."""
import time

import numpy as np
import pytest
import torch

from rtgb import abi, capi, scenes
from test_gpu_trace import _render_both
from test_gpu_wide import _grid_scene, _samples

pytestmark = pytest.mark.gpu


def compare_both_sides(ctx, orc, sc, smp, min_leaf=1):
    """The samples as they are (four lanes per ray) and repeated past 768 per SM (one
    lane per ray); the oracle traces them once.  Returns the number of hits."""
    n = smp.shape[0]
    line = 768 * torch.cuda.get_device_properties(0).multi_processor_count
    assert n <= line
    g, o = capi.Scene(ctx, sc), orc.new_scene(sc)
    g.build(30, min_leaf)
    o.build(30, min_leaf, 0)
    ref = o.trace(smp)
    o.shadow(smp, ref)
    hit = ref["hit"] == 1
    for total in (n, line + 1):
        k = np.arange(total) % n
        smp_d, hit_d = ctx.to_device(smp[k]), ctx.alloc(64 * total)
        hit_d.zero()
        g.trace(smp_d, total, hit_d)
        g.shadow(smp_d, total, hit_d)
        ctx.sync()
        got, m = hit_d.read(abi.HIT_DTYPE), hit[k]
        assert np.array_equal(got["hit"], ref["hit"][k])
        for f in ("id", "t", "inverse_n", "shadow_hit"):
            assert np.array_equal(got[f][m], ref[f][k][m]), (f, total)
        for f in ("n", "hit_point"):
            assert np.array_equal(got[f][m][:, :3], ref[f][k][m][:, :3]), (f, total)
    assert ctx.device_status() == 0
    return int(hit.sum())


def _axis_rays(n, seed, lo, hi, step):
    """Origins on a lattice (on box faces), directions with one or two zero
    components of either sign; every seventh ray ordinary."""
    r = np.random.default_rng(seed)
    lo, hi = np.array(lo), np.array(hi)
    o = (r.integers(lo / step, hi / step + 1, (n, 3)) * step).astype(np.float32)
    d = r.choice(np.array([-1.0, -0.0, 0.0, 1.0, 0.5], np.float32), (n, 3))
    d[(d == 0).all(axis=1)] = (0.0, -1.0, 0.0)
    d[::7] = r.normal(size=d[::7].shape)
    return _samples(o, d)


def _blocks(light_dir, seed=6):
    """Cubes of whole sizes on whole places: every leaf's box is flat."""
    r = np.random.default_rng(seed)
    corners = np.array([[x, y, z] for x in (0, 1) for y in (0, 1) for z in (0, 1)], np.float32)
    faces = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    pos, nrm, idx = [], [], []
    for _ in range(120):
        c = corners * r.integers(1, 4, 3) + r.integers(0, 14, 3)
        mid = c.mean(0)
        for f in faces:
            q = c[list(f)].astype(np.float32)
            n = q.mean(0) - mid
            k = 4 * len(pos)
            pos.append(q)
            nrm.append(np.tile(n / np.linalg.norm(n), (4, 1)))
            idx += [k, k + 1, k + 2, k, k + 2, k + 3]
    pad = lambda v: np.pad(np.concatenate(v).astype(np.float32), ((0, 0), (0, 1)))  # noqa: E731
    mats = np.zeros(1, abi.MATERIAL_DTYPE)
    mats["texture"], mats["diffuse"] = -1, 0.5
    lights = abi.make_lights((0.1,) * 3, [dict(type=abi.RT_DIR_L, dir=light_dir),
                                          dict(type=abi.RT_POINT_L, pos=(7.0, 30.0, 7.0))])
    return scenes.Scene(pad(pos), pad(nrm), np.array(idx, np.uint32), mats,
                        np.zeros(len(idx) // 3, np.uint32), lights)


DIRS = [(0.0, -1.0, 0.0), (-1.0, -0.0, 0.0), (0.0, -0.6, 0.8)]


@pytest.mark.parametrize("light_dir", DIRS)
@pytest.mark.parametrize("tmax", [1e37, np.inf])
def test_height_field_on_whole_numbers(ctx, orc, light_dir, tmax):
    smp = _axis_rays(8192, 8, (-1, -4, -1), (25, 5, 25), 1.0)
    smp["tmax"][::2] = tmax
    assert compare_both_sides(ctx, orc, _grid_scene(light_dir), smp) > 500


@pytest.mark.parametrize("light_dir", DIRS)
@pytest.mark.parametrize("tmax", [1e37, np.inf])
@pytest.mark.parametrize("min_leaf", [1, 9])
def test_flat_boxes_in_the_ray_s_plane(ctx, orc, light_dir, tmax, min_leaf):
    smp = _axis_rays(8192, 9, (-2, -2, -2), (18, 18, 18), 0.5)
    smp["tmax"][1::2] = tmax
    assert compare_both_sides(ctx, orc, _blocks(light_dir), smp, min_leaf) > 2000


def test_bounds_and_origins_at_infinity(ctx, orc):
    """Every combination of a bound or an origin that no slab can order, over
    parallel and ordinary directions, among rays without one."""
    smp = _axis_rays(8192, 10, (-2, -2, -2), (18, 18, 18), 0.5)
    r = np.random.default_rng(11)
    kind = r.integers(0, 9, smp.shape[0])
    inf, nan = np.float32(np.inf), np.float32(np.nan)
    smp["tmax"][(kind == 1) | (kind == 2)] = inf
    smp["tmin"][(kind == 2) | (kind == 3)] = -inf
    for k, v in ((4, inf), (5, -inf), (6, nan)):
        for a in range(3):
            smp["ori"][(kind == k) & (r.integers(0, 3, smp.shape[0]) == a), a] = v
    smp["inv_dir"][kind == 7, :3] = 1e-7   # no axis that counts
    neg = kind == 8                        # all components below zero, no lower bound
    smp["dir"][neg, :3] = -np.abs(smp["dir"][neg, :3]) - np.float32(0.25)
    smp["inv_dir"][neg, :3] = np.float32(1) / smp["dir"][neg, :3]
    smp["tmin"][neg] = -inf
    assert compare_both_sides(ctx, orc, _blocks(DIRS[2]), smp) > 1000


@pytest.mark.parametrize("light_dir", DIRS)
@pytest.mark.parametrize("w,h", [(150, 97), (401, 397)])
def test_frames_under_parallel_lights(ctx, orc, light_dir, w, h):
    """The fused renders, on both sides of the line: every pixel of a field of
    blocks with mirrors, lit along an axis or in a plane of two."""
    sc = _blocks(light_dir)
    sc.mats["reflectiveness"] = 0.4
    cam = scenes.camera((7.0, 26.0, -9.0), (7.0, 3.0, 7.0), aspect=w / h)
    img, _, st, rimg, rst, _, _ = _render_both(ctx, orc, sc, cam, w, h, 3)
    assert np.array_equal(img, rimg)
    assert (st[0], st[1], st[2], st[3]) == (rst.primary_rays, rst.secondary_rays, rst.shadow_rays, rst.hits)
    assert rst.hits > 0 and ctx.device_status() == 0


@pytest.mark.parametrize("what", ["trace", "shadow"])
def test_parallel_rays_cost_no_more_than_tilted_ones(ctx, what):
    """2.1 million rays over a small mesh, where a search's steps are what counts:
    along an axis and a degree off it they cross the same boxes within a few
    per cent, and a search by binary levels takes 1.4 times as long or more."""
    side = 1448
    y, x = np.mgrid[0:side, 0:side].astype(np.float32) / side * 2 - 1
    best = {}
    for name, d in (("axis", (0.0, 0.0, 1.0)), ("tilted", (0.012, 0.009, 0.99989))):
        sc = scenes.soup(10000, seed=7)
        sc.lights = abi.make_lights((0.1,) * 3, [dict(type=abi.RT_DIR_L, dir=d)])
        g = capi.Scene(ctx, sc)
        g.build(30, 1)
        o = np.stack([x.ravel(), y.ravel(), np.full(x.size, -4, np.float32)], 1)
        smp = _samples(o, np.tile(np.array(d, np.float32), (x.size, 1)))
        smp_d, hit_d = ctx.to_device(smp), ctx.alloc(64 * smp.shape[0])
        hit_d.zero()
        g.trace(smp_d, smp.shape[0], hit_d)
        run = (lambda: g.trace(smp_d, smp.shape[0], hit_d)) if what == "trace" else \
              (lambda: g.shadow(smp_d, smp.shape[0], hit_d))
        times = []
        for _ in range(15):
            ctx.sync()
            t = time.perf_counter()
            run()
            ctx.sync()
            times.append(time.perf_counter() - t)
        best[name] = min(times)
        g.close()
    assert best["axis"] < 1.25 * best["tilted"], best
