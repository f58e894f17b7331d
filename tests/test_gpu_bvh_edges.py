"""The GPU builder at the edges of its parts, byte for byte against the host builder: ranges of 255 to
258 items (one warp or one level), chunks of 256, levels whose ranges leave partly filled chunks,
sizes whose permutation bytes and shared arrays are full, and boxes whose infinities or zeros make
bounds, centroids and costs degenerate."""
import numpy as np
import pytest

from barnacle_gb300 import BarnacleError, bvh_build

pytestmark = pytest.mark.gpu


def same(ctx, boxes):
    hn, hp = bvh_build(boxes)
    dn, dp = ctx.bvh_build(boxes)
    assert hn.tobytes() == dn.tobytes() and np.array_equal(hp, dp)
    return hn


def cloud(n, seed, grid=None):
    rng = np.random.default_rng(seed)
    c = rng.normal(size=(n, 3)) * [40, 10, 40]
    if grid:
        c = np.round(c / grid) * grid
    h = np.exp(rng.normal(size=(n, 3)) * 0.7 - 2)
    return np.concatenate([c - h, c + h], 1).astype(np.float32)


@pytest.mark.parametrize("grid", [None, 8.0])
@pytest.mark.parametrize("n", [2, 3, 6, 31, 33, 255, 256, 257, 258, 511, 512, 513, 769, 1025, 4097, 66001, 300007])
def test_sizes(ctx, n, grid):
    same(ctx, cloud(n, n, grid))


@pytest.mark.parametrize("n", [200, 700, 20000])
def test_degenerate_boxes(ctx, n):
    rng = np.random.default_rng(n)
    t = rng.uniform(-1, 1, n).astype(np.float32)
    flat = np.zeros((n, 6), np.float32)
    flat[:, 0] = flat[:, 3] = t                       # points on a line: every area is zero
    flat[:, 1:3] = np.where(rng.random((n, 2)) < 0.5, 0.0, -0.0)
    flat[:, 4:6] = np.where(rng.random((n, 2)) < 0.5, 0.0, -0.0)
    same(ctx, flat)
    huge = cloud(n, 3) * np.float32(1e36)             # areas and costs overflow to infinity
    same(ctx, huge)
    up = cloud(n, 4)
    up[:, 3] = np.inf                                 # every x centroid infinite: the extent is NaN
    same(ctx, up)
    all_x = cloud(n, 5)
    all_x[n // 2, 0], all_x[n // 2, 3] = -np.inf, np.inf  # no centroid: the host builder's fold decides
    try:
        bvh_build(all_x)
    except BarnacleError:
        with pytest.raises(BarnacleError):
            ctx.bvh_build(all_x)
    else:
        same(ctx, all_x)


def test_small_input_with_an_infinite_box_is_refused_or_fits(ctx):
    b = cloud(100, 6)
    b[7, 3] = np.inf
    assert len(same(ctx, b)) == 129
    small = cloud(10, 7)
    small[2, 3] = np.inf                              # 129 nodes do not fit 2 n = 20
    with pytest.raises(BarnacleError):
        ctx.bvh_build(small)


def test_builds_of_changing_sizes_share_one_workspace(ctx):
    for n in (5000, 40, 90000, 257, 3, 5000):
        same(ctx, cloud(n, n + 1))
