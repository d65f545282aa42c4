"""The default render configuration is a choice by the frame's size with a number
of its own: a kernel that a caller names is the one that runs, and reading the
configuration and setting it again changes nothing."""
import numpy as np
import pytest

from rtgb import capi, scenes

pytestmark = pytest.mark.gpu

QUAD, AUTO = -2, -1   # from the end: four lanes per pixel, by the frame's size


def test_the_default_is_no_kernel_of_its_own(ctx, orc):
    c = capi.Context(0)
    sc = scenes.soup(3000, seed=14)
    g, o = capi.Scene(c, sc), orc.new_scene(sc)
    g.build(30, 1)
    o.build(30, 1, 0)
    infos = c.variants()
    first = c.render_config()
    assert first.variant == len(infos) + AUTO and first.blocks_per_sm == 0
    pooled = [v for v in range(len(infos) + QUAD) if infos[v] == infos[AUTO] and c.variant_pooled(v)]
    assert len(pooled) == 1   # the kernel of large frames has its own number too
    for w, h in ((192, 192), (401, 397)):   # on both sides of the line
        cam = scenes.camera((0.0, 0.0, -4.0), (0.0, 0.0, 0.0), aspect=w / h)
        ref, _ = o.render(cam, w, h, 3)
        rgba, img = c.alloc(4 * w * h), c.alloc(12 * w * h)
        for v, blocks in ((pooled[0], 0), (pooled[0], 2), (len(infos) + QUAD, 0), (first.variant, 0), (first.variant, 3)):
            c.set_render_config(v, blocks, first.chunk)
            got = c.render_config()
            assert (got.variant, got.blocks_per_sm, got.chunk) == (v, blocks, first.chunk)
            g.render(cam, w, h, 3, rgba, img)
            c.sync()
            assert np.array_equal(img.read(np.uint32).reshape(-1, 3), ref), (v, blocks, w)
        cfg, _ = g.autotune(cam, w, h, 3, trials=1)
        assert cfg.variant != first.variant   # the tuner names a kernel
    assert c.device_status() == 0
    g.close()
    c.close()
