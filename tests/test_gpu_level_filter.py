"""The level form's first-level filter (levels.cu, lv_filter_full) at the edges
of its packs of four and eight candidates, its steps of 8,192 and its staging,
with few candidates (fewer than pruners) and many in an attribute's lowest
cell: the level form forced, against the bitmap form on every cuboid."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen

pytestmark = pytest.mark.gpu


def same(ctx, x, max_d):
    d = x.shape[1]
    ds = sk.Dataset(ctx, x)
    a = sk.skycube(ctx, ds, max_d=max_d, want_extended=True, form="levels")
    b = sk.skycube(ctx, ds, max_d=max_d, want_extended=True, form="bitmaps")
    assert a.form()[0] == "levels"
    for c in range(1, 1 << d):
        assert np.array_equal(a.cuboid(c), b.cuboid(c)), (x.shape, max_d, c)
        assert np.array_equal(a.extended(c), b.extended(c)), (x.shape, max_d, c)
    assert a.info()["total_skyline_ids"] == b.info()["total_skyline_ids"]
    for o in (a, b, ds):
        o.close()


@pytest.mark.parametrize("n", [1, 3, 4, 5, 7, 8, 9, 63, 65, 8191, 8192, 8193, 16385, 24577])
@pytest.mark.parametrize("d,max_d", [(3, 1), (6, 4), (9, 2)])
def test_candidate_counts(gpu_ctx, n, d, max_d):
    x = np.random.default_rng(n).random((n, d), dtype=np.float32)
    x[:, 0] = d - x[:, 1:].sum(axis=1)  # every point is a candidate
    same(gpu_ctx, x, max_d)


@pytest.mark.parametrize("max_d", [1, 2, 3, 4])
def test_crowded_lowest_cells(gpu_ctx, max_d):
    x = datagen.generate("anticorrelated", 20000, 7, 3)
    x[: 2000] *= 0.001  # strong points crowd the lowest cells
    x[:, 3] = np.float32(0.25) - x[:, 3] * np.float32(0.25)
    same(gpu_ctx, x, max_d)
