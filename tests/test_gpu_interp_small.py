"""Small host calls of the GPU interpolator: queries spread thinly over warps, and arrays that
go up and down in one block, at the edges of both rules.  The bits are the host queries'."""
import numpy as np
import pytest

from fastlem_gb300.api import TerrainInterpolator2D

pytestmark = pytest.mark.gpu

WARPS = 152 * 12                      # blocks that a small batch is spread over
BLOCK = 1 << 20                       # bytes of the block


def fits(n):
    """The largest batch over n sites that goes through the block."""
    return (BLOCK - 64 - 4 - 8 * n) // 29


@pytest.mark.parametrize("n, count", [
    (3, 1), (3, WARPS), (500, WARPS + 1), (500, 2 * WARPS + 7),
    (2_000, fits(2_000)), (2_000, fits(2_000) + 1), (400, 32 * WARPS), (400, 32 * WARPS + 1),
    ((BLOCK - 64 - 4 - 29) // 8, 1), ((BLOCK - 64 - 4) // 8 + 1, 1)])
def test_small_calls_same_bits(n, count):
    r = np.random.default_rng(n + count)
    if n == 2_000:                    # a lattice: sites on shared circles, many deferred queries
        gx, gy = np.meshgrid(np.arange(50.0), np.arange(40.0))
        xs, ys = gx.ravel(), gy.ravel()
        qx, qy = r.integers(-2, 100, count) / 2.0, r.integers(-2, 80, count) / 2.0
    else:
        xs, ys = r.uniform(0, 50, n), r.uniform(0, 40, n)
        qx, qy = r.uniform(-2, 52, count), r.uniform(-2, 42, count)
    it = TerrainInterpolator2D(xs, ys)
    for seed in (1, 2):               # the second call over what the first left
        f = np.random.default_rng(seed).normal(0, 1, n)
        host, hok = it.interpolate_many(f, qx, qy)
        dev, dok = it.interpolate_many(f, qx, qy, gpu=True)
        assert np.array_equal(hok, dok)
        assert np.array_equal(host.view(np.uint64), dev.view(np.uint64))
        qx, qy = qx[::-1].copy(), qy[::-1].copy()
