"""The autotuner over frames that no variant may follow for ever: mirrors that
face each other on all sides, at depths past what rt_render takes."""
import numpy as np
import pytest

from rtgb import abi, capi, scenes

pytestmark = pytest.mark.gpu


def _mirror_cube():
    """Inside of a cube, every face a full mirror: a path never leaves it."""
    corners = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32)
    faces = [(0, 1, 3, 2), (4, 6, 7, 5), (0, 4, 5, 1), (2, 3, 7, 6), (0, 2, 6, 4), (1, 5, 7, 3)]
    pos, nrm, idx = [], [], []
    for f in faces:
        q = corners[list(f)]
        n = -q.mean(0)
        k = len(pos) * 4
        pos.append(q)
        nrm.append(np.tile(n, (4, 1)))
        idx += [k, k + 1, k + 2, k, k + 2, k + 3]
    pad = lambda v: np.pad(np.concatenate(v).astype(np.float32), ((0, 0), (0, 1)))
    mats = np.zeros(1, abi.MATERIAL_DTYPE)
    mats["texture"], mats["diffuse"], mats["reflectiveness"] = -1, 0.5, 1.0
    lights = abi.make_lights((0.1,) * 3, [dict(type=abi.RT_POINT_L, pos=(0.3, 0.2, 0.1))])
    return scenes.Scene(pad(pos), pad(nrm), np.array(idx, np.uint32), mats, np.zeros(12, np.uint32), lights)


@pytest.mark.parametrize("bounces", [-1, 255, 256, 300])
def test_autotune_depth_is_bounded(ctx, bounces):
    g = capi.Scene(ctx, _mirror_cube())
    g.build(30, 1)
    saved = ctx.render_config()
    cam = scenes.camera((0.1, 0.2, -0.5), (0.0, 0.1, 0.5))
    cfg, _ = g.autotune(cam, 40, 24, bounces, trials=1)
    assert 0 <= cfg.variant < len(ctx.variants())
    ctx.set_render_config(saved.variant, saved.blocks_per_sm, saved.chunk)
    assert ctx.device_status() == 0
    g.close()


def test_autotune_reports_the_chunk_in_use(ctx):
    """The kernel with four lanes per pixel shares a frame out by its size: the
    tuner tries it with one chunk and reports that one."""
    g = capi.Scene(ctx, scenes.soup(3000, seed=8))
    g.build(30, 1)
    saved = ctx.render_config()
    quad = len(ctx.variants()) - 2   # the last one is the choice by the frame's size
    for w, h in ((16, 16), (40, 24), (64, 64)):
        cfg, ms = g.autotune(scenes.camera((0, 0, -4), (0, 0, 0), aspect=w / h), w, h, 3, trials=5)
        assert ms > 0 and (cfg.variant != quad or cfg.chunk == 32)
    ctx.set_render_config(saved.variant, saved.blocks_per_sm, saved.chunk)
    g.close()
