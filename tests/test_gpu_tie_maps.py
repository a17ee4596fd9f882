"""The bitmap kernel's tie maps (mdmc.cu) where many float ties meet: points of
one coordinate sum on a coarse integer grid (none dominates another on the
full space, so every point is a q and ties with most others), in shared
memory (11 attributes), as a list and in the global slab, closed in registers
(12 and more); per-point bitmaps against their definition, and capped runs
(the closure over 1 to 64 rows) against the uncapped bits."""
import itertools

import numpy as np
import pytest

import oracle
import skycube_gb300 as sk

pytestmark = pytest.mark.gpu


def tied_points(n, d, levels, seed):
    x = np.random.default_rng(seed).integers(0, levels, size=(n, d)).astype(np.float32)
    x[:, 0] = levels * d - x[:, 1:].sum(axis=1)
    return x


def brute_bits(x):
    n, d = x.shape
    S = np.arange(1 << d, dtype=np.uint32)
    w = (1 << np.arange(d)).astype(np.uint32)
    out = np.zeros((n, 1 << d), dtype=bool)
    for p in range(n):
        le = np.unique((((x <= x[p]) @ w).astype(np.uint64) << np.uint64(32)) |
                       ((x < x[p]) @ w).astype(np.uint64))
        for e in le:
            E, L = np.uint32(int(e) >> 32), np.uint32(int(e) & 0xffffffff)
            if L:
                out[p] |= ((S & ~E) == 0) & ((S & L) != 0)
    return out


@pytest.mark.parametrize("d,n,levels", [(10, 150, 3), (11, 120, 3), (12, 100, 2), (12, 90, 4),
                                        (13, 70, 3), (14, 50, 2), (16, 40, 3), (16, 20, 9)])
def test_bitmaps_with_many_ties(gpu_ctx, d, n, levels):
    x = tied_points(n, d, levels, 100 * d + n)
    ds = sk.Dataset(gpu_ctx, x)
    r = sk.skycube(gpu_ctx, ds, want_bitmaps=True)
    bits, pids = r.bitmaps()
    assert np.array_equal(pids, np.arange(n))
    got = ((bits[:, :, None] >> np.arange(32, dtype=np.uint32)) & 1).reshape(n, -1).astype(bool)
    want = brute_bits(x)
    assert np.array_equal(got[:, : 1 << d], want)
    for cap in (1, 3, 6, d - 2):
        a = sk.skycube(gpu_ctx, ds, max_d=cap, form="bitmaps")
        for c in range(1, 1 << d, 7 if d < 14 else 61):
            ids = a.cuboid(c)
            if bin(c).count("1") <= cap or c == (1 << d) - 1:
                assert np.array_equal(ids, np.flatnonzero(~want[:, c])), (d, cap, c)
            else:
                assert len(ids) == 0
        a.close()
    r.close()
    ds.close()


def tie_pairs(d, k, covered, seed):
    """A point p (index 0) that ties with k points on 6 attributes each, below
    it on one of those and above it on the others: k maximal (LE, LT) pairs,
    and `covered` points more whose 5 or 4 attributes lie inside one of them."""
    rng = np.random.default_rng(seed)
    sets = [c for c in itertools.islice(itertools.combinations(range(d), 6), 4000)]
    rows = [np.full(d, 5.0)]
    for i in rng.permutation(len(sets))[:k]:
        q = np.full(d, 6.0)
        q[list(sets[i])] = 5.0
        q[sets[i][rng.integers(6)]] = 4.0
        rows.append(q)
    for j in range(covered):
        q = rows[1 + j % k].copy()
        same = np.flatnonzero(q == 5.0)
        q[rng.choice(same, 1 + j % 2, replace=False)] = 6.5 + j
        rows.append(q)
    return np.array(rows, np.float32)


@pytest.mark.parametrize("d,max_d", [(12, 0), (13, 6), (16, 4)])
@pytest.mark.parametrize("k,covered", [(1, 40), (31, 30), (32, 0), (32, 90), (33, 0), (300, 50)])
def test_lists_of_maximal_pairs(gpu_ctx, d, max_d, k, covered):
    """A candidate's tie pairs above 11 attributes: maximal ones in a list of
    32, the global map from the 33rd on, pairs inside another dropped in
    whichever order they come; against the oracle."""
    x = tie_pairs(d, k, covered, 7 * k + d)
    order = np.random.default_rng(k).permutation(len(x))
    x = np.ascontiguousarray(x[order])
    sky, ext = oracle.stsc(x, max_d or d)
    ds = sk.Dataset(gpu_ctx, x)
    r = sk.skycube(gpu_ctx, ds, max_d=max_d, want_extended=True, form="bitmaps")
    for c in sky:
        assert np.array_equal(r.cuboid(c), sky[c]), c
        assert np.array_equal(r.extended(c), ext[c]), c
    r.close()
    ds.close()
