"""The skyline kernel's box tree (partition.cu, k_skyline_tree) against
brute-force statuses: sizes around the edges of its groups of 32 points,
quarters, halves and padded last block, lists long enough that an item is
cut into slices, ties at the attributes' minima (its two early exits), equal
points, signed zeros, coarse grids, and subspaces of 1 to 16 attributes."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen

pytestmark = pytest.mark.gpu


def brute(x):
    sky, ext = [], []
    for p in range(len(x)):
        le = x <= x[p]
        lt = x < x[p]
        dom = le.all(axis=1) & lt.any(axis=1)
        if not dom.any():
            sky.append(p)
        elif not lt.all(axis=1).any():
            ext.append(p)
    return np.array(sky, np.uint32), np.array(ext, np.uint32)


def check(ctx, x, subspaces, **opts):
    ds = sk.Dataset(ctx, x)
    for S in subspaces:
        cols = [k for k in range(x.shape[1]) if S >> k & 1]
        sky, ext = brute(x[:, cols])
        r = sk.skycube(ctx, ds, subspace=S, **opts)
        assert np.array_equal(r.cuboid(S), sky), (x.shape, S, opts)
        assert np.array_equal(r.extended(S), ext), (x.shape, S, opts)
        r.close()
    ds.close()


@pytest.mark.parametrize("n", [1, 2, 7, 8, 31, 32, 33, 63, 65, 255, 257, 1025])
def test_edges_of_groups_and_blocks(gpu_ctx, n):
    for kind, d in (("anticorrelated", 5), ("ties", 3), ("uniform", 9)):
        x = datagen.generate(kind, n, d, 100 + n)
        check(gpu_ctx, x, [(1 << d) - 1, 0b101, 0b10])


@pytest.mark.parametrize("kind,n,d", [("anticorrelated", 9001, 12), ("uniform", 7000, 4),
                                      ("ties", 6000, 10), ("correlated_q", 5000, 16),
                                      ("anticorrelated", 4097, 16)])
@pytest.mark.parametrize("pq_size", [-1, 64])
def test_slices_and_wide_subspaces(gpu_ctx, kind, n, d, pq_size):
    x = datagen.generate(kind, n, d, 7)
    full = (1 << d) - 1
    check(gpu_ctx, x, [full, full >> 1, full & 0x5555, 0b11], pq_size=pq_size)


@pytest.mark.parametrize("depth", [1, 2, 7])
def test_minima_duplicates_and_signed_zeros(gpu_ctx, depth):
    rng = np.random.default_rng(depth)
    x = rng.integers(0, 4, size=(3000, 6)).astype(np.float32)
    x[::5] = x[0]                      # many equal points
    x[x == 0] *= rng.choice([-1.0, 1.0], size=(x == 0).sum()).astype(np.float32)
    check(gpu_ctx, x, [63, 0b111, 0b100100, 0b1], depth=depth)
    same = np.full((100, 4), 2.5, np.float32)
    check(gpu_ctx, same, [15, 0b110], depth=depth)
