"""The tree and leaf sizes of the four-wide records' tests on both sides of the
line between four lanes and one lane per ray (a launch of few rays never reaches
the one-lane search of the stage kernels), and boxes with NaN corners."""
import numpy as np
import pytest

from helpers import tiny_terrain
from rtgb import scenes
from test_gpu_careful import _axis_rays, compare_both_sides
from test_gpu_wide import _random_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,min_leaf", [(1, 1), (2, 1), (3, 1), (4, 1), (5, 1), (5, 4), (6, 4), (7, 1), (9, 1), (16, 4),
                                        (33, 1), (257, 1), (300, 5), (300, 8), (300, 9), (511, 256), (512, 1), (513, 1),
                                        (2000, 64), (4097, 2), (4609, 1), (40000, 1)])
def test_trees_and_leaves_of_every_size(ctx, orc, n, min_leaf):
    sc = scenes.soup(n, seed=n, offset_sigma=max(0.03, 0.5 / n ** 0.4))
    assert compare_both_sides(ctx, orc, sc, _random_rays(4001, n), min_leaf) > 0


@pytest.mark.parametrize("axis", [0, 1, 2, 3])
def test_nan_vertices(ctx, orc, axis):
    """Vertices with a NaN coordinate (3: all of them): a triangle of such a vertex is
    never hit, its neighbours are."""
    sc = tiny_terrain(48, 24, 4).scene(2)
    sc.pos4 = sc.pos4.copy()
    bad = np.random.default_rng(13).random(sc.n_verts) < 0.05
    sc.pos4[bad, slice(0, 3) if axis == 3 else axis] = np.nan
    smp = _axis_rays(8000, 14, (-8, -2, -4), (8, 6, 4), 0.25)
    half = _random_rays(4000, 15)
    smp["ori"][::2, :3] = half["ori"][:, :3] * np.float32(3)
    smp["dir"][::2], smp["inv_dir"][::2] = half["dir"], half["inv_dir"]
    assert compare_both_sides(ctx, orc, sc, smp) > 300
