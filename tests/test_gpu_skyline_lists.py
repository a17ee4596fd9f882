"""Lists past the short-list kernel's limit (small.cu, 6,144 points) through
the skyline kernel (partition.cu, k_skyline_tree) without a prefilter, so that
nothing else settles them: sizes around the edges of its groups, quarters,
halves and padded last block, subspace lists of 1 to 16 attributes, slices,
ties at the minima with equal points and signed zeros. Every call is checked to
take that kernel; statuses against brute force."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen

pytestmark = pytest.mark.gpu

SHORT = 6144  # kSmallList


def statuses(x):
    """Skyline and extended skyline ids by brute force."""
    st = np.empty(len(x), np.uint8)
    for b in range(0, len(x), 256):
        p = x[b:b + 256]
        le = np.ones((len(p), len(x)), bool)
        lt_all, lt_any = le.copy(), np.zeros_like(le)
        for k in range(x.shape[1]):
            lt = x[None, :, k] < p[:, None, k]
            le &= x[None, :, k] <= p[:, None, k]
            lt_all &= lt
            lt_any |= lt
        st[b:b + 256] = np.where(lt_all.any(axis=1), 2, np.where((le & lt_any).any(axis=1), 1, 0))
    return np.flatnonzero(st == 0), np.flatnonzero(st == 1)


def check(ctx, x, subspaces, **opts):
    d = x.shape[1]
    full = (1 << d) - 1
    ds = sk.Dataset(ctx, x)
    for S in subspaces:
        r = sk.skycube(ctx, ds, subspace=S, **opts)
        names = [p for p, _ in ctx.last_phases()]
        assert "full: pivots+cells" in names and "full: prefilter" not in names
        assert S == full or r.info()["n_candidates"] > SHORT
        sky, ext = statuses(x[:, [k for k in range(d) if S >> k & 1]])
        assert np.array_equal(r.cuboid(S), sky), (x.shape, S)
        assert np.array_equal(r.extended(S), ext), (x.shape, S)
        r.close()
    ds.close()


def plane(n, d, seed):
    """Points of a plane: all of them candidates, so that a subspace's list is
    as long as the data set."""
    x = np.random.default_rng(seed).random((n, d), dtype=np.float32)
    x[:, 0] = d - x[:, 1:].sum(axis=1)
    return x


EDGES = [6145, 6146, 6147, 6148, 6149, 6151, 6152, 6153, 6159, 6160, 6161, 6175, 6176, 6177]


@pytest.mark.parametrize("n", EDGES)
def test_edges_of_groups_and_blocks(gpu_ctx, n):
    check(gpu_ctx, plane(n, 5, n), [31, 0b110, 0b10100, 0b1], pq_size=-1)
    check(gpu_ctx, datagen.generate("ties", n, 3, n), [7], pq_size=-1)
    check(gpu_ctx, datagen.generate("anticorrelated", n, 9, n), [511], pq_size=-1)


@pytest.mark.parametrize("n,d", [(6177, 2), (9001, 8), (16001, 12), (6500, 16)])
def test_subspaces_and_slices(gpu_ctx, n, d):
    full = (1 << d) - 1
    x = plane(n, d, d)
    subspaces = {full, full >> 1, full & 0x5555, 0b11, 0b10, full & ~0b100 if d > 2 else 1}
    check(gpu_ctx, x, sorted(subspaces), pq_size=-1)
    check(gpu_ctx, datagen.generate("uniform", n, d, 7), [full], pq_size=-1)


@pytest.mark.parametrize("seed", [1, 2, 7])
def test_minima_duplicates_and_signed_zeros(gpu_ctx, seed):
    rng = np.random.default_rng(seed)
    x = rng.integers(0, 4, size=(9000, 6)).astype(np.float32)
    x[::5] = x[0]                      # many equal points
    x[x == 0] *= rng.choice([-1.0, 1.0], size=(x == 0).sum()).astype(np.float32)
    check(gpu_ctx, x, [63], pq_size=-1)
    x = plane(7000, 6, seed)           # candidates on every subspace, with the minima tied
    x[:, 1:] = np.floor(x[:, 1:] * 3)
    x[:, 0] = 20 - x[:, 1:].sum(axis=1)
    x[x == 0] *= rng.choice([-1.0, 1.0], size=(x == 0).sum()).astype(np.float32)
    check(gpu_ctx, x, [63, 0b111, 0b100100, 0b10, 0b111110], pq_size=-1)
    check(gpu_ctx, np.full((6200, 4), 2.5, np.float32), [15, 0b110], pq_size=-1)
