"""Coarse grids asked for by the caller (depth 1 and 2): results never depend
on the depth, and neither does the cost of the steps whose kernels live on fine
cells. On two cells per attribute nearly every pair of points ties, so the
skyline kernel, which reads tied floats by point id, was 20 times as slow as on
the default grid; it, the prefilter and the subspace skylines use that grid at
any depth. Bounds are ratios of device times of the same call, far from 1
before and within noise of it now."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen

pytestmark = pytest.mark.gpu


def device_ms(ctx, ds, reps=4, **opts):
    best = float("inf")
    for _ in range(reps):
        r = sk.skycube(ctx, ds, **opts)
        best = min(best, ctx.last_device_ms())
        r.close()
    return best


@pytest.mark.parametrize("kind,n,d,S", [("uniform", 300000, 10, 0b1010110100),
                                        ("anticorrelated", 200000, 8, 0b11111111)])
@pytest.mark.parametrize("depth", [1, 2])
def test_skyline_queries_cost_the_same(gpu_ctx, kind, n, d, S, depth):
    ds = sk.Dataset(gpu_ctx, datagen.generate(kind, n, d, 4))
    a = sk.skycube(gpu_ctx, ds, subspace=S)
    b = sk.skycube(gpu_ctx, ds, subspace=S, depth=depth)
    assert np.array_equal(a.cuboid(S), b.cuboid(S))
    assert np.array_equal(a.extended(S), b.extended(S))
    for o in (a, b):
        o.close()
    assert device_ms(gpu_ctx, ds, subspace=S, depth=depth) < 2 * device_ms(gpu_ctx, ds, subspace=S)
    ds.close()


@pytest.mark.parametrize("kind,n,d,max_d", [("anticorrelated", 200000, 12, 3), ("uniform", 300000, 12, 4)])
@pytest.mark.parametrize("depth", [1, 2])
def test_level_form_costs_the_same(gpu_ctx, kind, n, d, max_d, depth):
    """The level form's first-level filter drops by cells alone, so on two
    cells per attribute it dropped next to nothing (23 ms against 1.0 at 200k x
    12, and past the survivors' capacity at 500k x 16 the whole launch was
    thrown away); its grid is its own."""
    ds = sk.Dataset(gpu_ctx, datagen.generate(kind, n, d, 4))
    a = sk.skycube(gpu_ctx, ds, max_d=max_d, form="levels")
    b = sk.skycube(gpu_ctx, ds, max_d=max_d, form="levels", depth=depth)
    assert a.form() == b.form() == ("levels", 0)
    for c in range(1, 1 << d):
        if bin(c).count("1") <= max_d:
            assert np.array_equal(a.cuboid(c), b.cuboid(c)), c
    for o in (a, b):
        o.close()
    opts = {"max_d": max_d, "form": "levels"}
    assert device_ms(gpu_ctx, ds, depth=depth, **opts) < 2 * device_ms(gpu_ctx, ds, **opts)
    ds.close()


@pytest.mark.parametrize("kind,n,d,tile_points", [("uniform", 300000, 10, 65536),
                                                  ("anticorrelated", 200000, 8, 65536)])
def test_bitmap_order_on_two_cells(gpu_ctx, kind, n, d, tile_points):
    """A grid of two cells has no bits below the median's, and a q order
    without them leaves the partitions unsorted: the bitmap kernel took 3.4
    and 4.4 times as long as on four cells, in order of strength 2.7 and 3.5."""
    ds = sk.Dataset(gpu_ctx, datagen.generate(kind, n, d, 4))

    def kernel_ms(depth):
        best = float("inf")
        for _ in range(4):
            sk.skycube(gpu_ctx, ds, depth=depth, tile_points=tile_points).close()
            best = min(best, dict(gpu_ctx.last_phases())["bitmap kernel"])
        return best

    assert kernel_ms(1) < {"uniform": 3.0, "anticorrelated": 3.85}[kind] * kernel_ms(2)
    ds.close()
