"""Lists full of equal points through the skyline kernel (partition.cu): copies
of a point are left out of its boxes (repeats_earlier), across blocks, beside
other points' copies in one bucket, and not where only the cells are equal.
Statuses against those of the distinct points, which decide them."""
import numpy as np
import pytest

import skycube_gb300 as sk

pytestmark = pytest.mark.gpu


def expected(x):
    """Skyline and extended skyline ids, by brute force over the distinct rows
    (signed zeros are equal)."""
    u, inv = np.unique(x + np.float32(0), axis=0, return_inverse=True)
    st = np.zeros(len(u), np.uint8)
    for p in range(len(u)):
        le = (u <= u[p]).all(axis=1)
        le[p] = False
        if le.any():
            st[p] = 2 if (u[le] < u[p]).all(axis=1).any() else 1
    st = st[inv.ravel()]
    return np.flatnonzero(st == 0), np.flatnonzero(st == 1)


def check(ctx, x, subspaces, **opts):
    ds = sk.Dataset(ctx, x)
    for S in subspaces:
        sky, ext = expected(x[:, [k for k in range(x.shape[1]) if S >> k & 1]])
        r = sk.skycube(ctx, ds, subspace=S, **opts)
        assert any(p == "full: pivots+cells" for p, _ in ctx.last_phases())  # not the short-list kernel
        assert np.array_equal(r.cuboid(S), sky), (x.shape, S, opts)
        assert np.array_equal(r.extended(S), ext), (x.shape, S, opts)
        r.close()
    ds.close()


def grid(levels, n, d, seed):
    """Whole numbers, the points below a plane mirrored: many copies of every
    point, most of them not strictly dominated."""
    rng = np.random.default_rng(seed)
    x = rng.integers(0, levels, (n, d))
    low = x.sum(axis=1) < 0.4 * (levels - 1) * d
    x[low] = levels - 1 - x[low]
    return x.astype(np.float32)


@pytest.mark.parametrize("levels", [2, 3, 4, 7])
@pytest.mark.parametrize("n,d", [(6145, 4), (9001, 6), (20011, 5), (6177, 16), (7000, 2)])
def test_grids(gpu_ctx, levels, n, d):
    x = grid(levels, n, d, n + levels)
    full = (1 << d) - 1
    check(gpu_ctx, x, sorted({full, full & 0b101101101101101, full & 0b110, 1}), pq_size=-1)
    check(gpu_ctx, x, [full], pq_size=8)


def test_equal_cells_are_not_equal_points(gpu_ctx):
    """Points along a diagonal, 70 to a cell, three copies of each: repeats and
    other points with the same cells side by side; some differ by the zero's
    sign only."""
    rng = np.random.default_rng(5)
    u = rng.random(3000).astype(np.float32)
    x = np.stack([u, 1 - u + np.float32(1e-5) * rng.random(3000).astype(np.float32)], axis=1)
    x[:40, 0] = 0
    x = np.concatenate([x, x, x])[rng.permutation(9000)]
    z = (x[:, 0] == 0) & (rng.random(9000) < 0.5)
    x[z, 0] = -0.0
    check(gpu_ctx, np.ascontiguousarray(x), [1, 2, 3], pq_size=-1)


@pytest.mark.parametrize("levels,former_ms", [(2, 18.8), (4, 4.95)])
def test_copies_cost_no_more_than_before(gpu_ctx, levels, former_ms):
    """The kernel that compared all points of a partition took 18.8 and 4.95 ms;
    the box tree with every copy in its boxes took up to 28.2 and 8.5."""
    ds = sk.Dataset(gpu_ctx, grid(levels, 200000, 6, 1))
    best = float("inf")
    for _ in range(3):
        sk.skycube(gpu_ctx, ds, subspace=63).close()
        best = min(best, dict(gpu_ctx.last_phases())["full: skyline kernel"])
    assert best < former_ms
    ds.close()
