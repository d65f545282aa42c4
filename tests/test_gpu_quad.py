"""GPU parity of the searches with four lanes per ray: ray and pixel counts
around the warp's shares and the line to one lane per ray, and leaves longer
than four triangles.  Every hit record, shadow mask and pixel equals the
oracle's bit for bit."""
import numpy as np
import pytest
import torch

from helpers import tiny_terrain
from rtgb import scenes
from test_gpu_trace import _render_both
from test_gpu_wide import _compare, _random_rays

pytestmark = pytest.mark.gpu


def _sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("per_sm,more", [(0, 1), (0, 7), (0, 33), (16, 0), (16, 1), (32, 1), (64, 1),
                                         (64, 5), (768, 0), (768, 1)])
def test_ray_counts(ctx, orc, per_sm, more):
    sc = scenes.soup(3000, seed=5)
    _compare(ctx, orc, sc, _random_rays(per_sm * _sms() + more, per_sm + more))


@pytest.mark.parametrize("n,min_leaf", [(1, 1), (2, 1), (5, 4), (300, 5), (300, 8), (300, 9), (2000, 64)])
def test_leaf_sizes(ctx, orc, n, min_leaf):
    sc = scenes.soup(n, seed=n, offset_sigma=max(0.03, 0.5 / n ** 0.4))
    _compare(ctx, orc, sc, _random_rays(3000, n), min_leaf)


@pytest.mark.parametrize("w,h,bounces", [(1, 1, 4), (7, 3, 4), (64, 76, 4), (69, 71, 0), (97, 101, 4), (139, 141, 4),
                                         (341, 342, 4), (342, 342, 2)])
def test_small_frames(ctx, orc, w, h, bounces):
    """Two lights, mirrors, sizes on both sides of each share and of the line."""
    sc = tiny_terrain(96, 48, 12).scene(3)
    cam = scenes.camera((0.0, 4.0, -10.0), (0.0, 0.0, 0.0), aspect=w / h)
    img, rgba, st, rimg, rst, _, _ = _render_both(ctx, orc, sc, cam, w, h, bounces)
    assert np.array_equal(img, rimg)
    assert (st[0], st[1], st[2], st[3]) == (rst.primary_rays, rst.secondary_rays, rst.shadow_rays, rst.hits)
    assert ctx.device_status() == 0
