"""GPU parity of the searches with four lanes per ray: ray counts around the
warp's shares and the line to one lane per ray, and leaves longer than four
triangles.  Every hit record and shadow mask equals the oracle's bit for bit."""
import numpy as np
import pytest
import torch

from rtgb import scenes
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
