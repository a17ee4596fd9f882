"""CPU model of the skyline kernel's rules (csrc/partition.cu): which boxes of
the sorted list a point walks (partitions under its median mask, cut into
slices, each but the first opened by the list's first block; copies of a point
left out of the boxes' minima), which pairs it then compares in floats, and the
early exits of points that hold an attribute's minimum. Against brute force, on
data with ties, copies, signed zeros and few cells, with a hash that tells the
copies apart and one that never does."""
import numpy as np
import pytest

from skycube_gb300 import datagen


def brute(x):
    st = np.zeros(len(x), int)
    for p in range(len(x)):
        le, lt = x <= x[p], x < x[p]
        if lt.all(axis=1).any():
            st[p] = 2
        elif (le.all(axis=1) & lt.any(axis=1)).any():
            st[p] = 1
    return st


def cells_of(x, depth):
    """Pivots strictly below the value, 2^depth - 1 order statistics."""
    n, d = x.shape
    P = (1 << depth) - 1
    c = np.zeros((n, d), int)
    for k in range(d):
        s = np.sort(x[:, k])
        piv = s[[(r + 1) * n // (P + 1) for r in range(P)]]
        c[:, k] = np.searchsorted(piv, x[:, k], side="left")
    return c


def left_out(x, cells, hashes):
    """repeats_earlier for every entry of the sorted list."""
    out = np.zeros(len(x), bool)
    for i in range(len(x)):
        b = i // 32
        block = range(32 * b, min(len(x), 32 * b + 32))
        same = [j for j in block if hashes[j] == hashes[i]]
        src = same[0]
        if b > 0 and i == src and len(same) > 1:
            prev = [j for j in range(32 * b - 32, 32 * b) if hashes[j] == hashes[i]]
            src = prev[0] if prev else src
        out[i] = src != i and (x[i] == x[src]).all()
    return out


def model(x, depth, B, splits, rng, degenerate):
    n, d = x.shape
    cells = cells_of(x, depth)
    top = cells[:, :B] >> (depth - 1)
    mask = (top << np.arange(B)).sum(axis=1)
    rank = {m: r for r, m in enumerate(sorted(range(1 << B), key=lambda m: (bin(m).count("1"), m)))}
    finer = [tuple(c & ((1 << (depth - 1)) - 1)) for c in cells]  # equal points: one bucket
    order = sorted(range(n), key=lambda i: (rank[mask[i]], finer[i], rng.random()))
    x, cells, mask = x[order], cells[order], mask[order]
    amin = x.min(axis=0)
    hashes = [0 if degenerate else hash(tuple(c)) for c in cells]
    box = np.where(left_out(x, cells, hashes)[:, None], 127, cells)
    starts = {m: [i for i in range(n) if mask[i] == m] for m in range(1 << B)}
    st = np.zeros(n, int)
    for p in range(n):
        n_min = int((x[p] == amin).sum())
        if n_min == d:
            continue
        parts = [starts[m] for m in sorted(rank, key=rank.get) if m & ~mask[p] == 0]
        under = [i for part in parts for i in part]
        for sp in range(splits):
            lo, hi = len(under) * sp // splits, len(under) * (sp + 1) // splits
            blocks = ([0] if sp else []) + sorted({i // 32 for i in under[lo:hi]})
            for b in blocks:
                for h in range(8):  # 4-q halves; a padded entry has cells of 127
                    qs = range(32 * b + 4 * h, min(n, 32 * b + 4 * h + 4))
                    if not len(qs) or not (box[list(qs)].min(axis=0) <= cells[p]).all():
                        continue
                    for q in qs:
                        if (cells[q] <= cells[p]).all() and (x[q] <= x[p]).all() and (x[q] < x[p]).any():
                            strict = (x[q] < x[p]).all()
                            assert not (strict and n_min)
                            st[p] |= 3 if strict else 1
    out = np.zeros(n, int)
    out[order] = np.where(st > 1, 2, st)
    return out


@pytest.mark.parametrize("kind,n,d,depth,B,splits,degenerate", [
    ("uniform", 150, 4, 3, 3, 1, False), ("anticorrelated", 130, 5, 7, 4, 3, False),
    ("ties", 160, 3, 7, 2, 2, False), ("grid", 200, 3, 7, 3, 1, False),
    ("grid", 200, 3, 7, 3, 4, False), ("grid", 161, 4, 2, 2, 2, False),
    ("grid", 190, 3, 7, 2, 3, True), ("copies", 192, 3, 7, 3, 2, False),
    ("copies", 193, 2, 3, 1, 3, True), ("uniform", 33, 2, 7, 2, 2, True)])
def test_model_against_brute_force(kind, n, d, depth, B, splits, degenerate):
    rng = np.random.default_rng(n + d + splits)
    for _ in range(3):
        if kind == "grid":
            x = rng.integers(0, 3, (n, d)).astype(np.float32)
            x[x.sum(axis=1) < d] = 2
            x[x == 0] *= rng.choice([-1.0, 1.0], size=(x == 0).sum()).astype(np.float32)
        elif kind == "copies":
            x = np.repeat(datagen.generate("anticorrelated", n // 6 + 1, d, 3), 6, axis=0)[:n]
            x = x[rng.permutation(n)]
        else:
            x = datagen.generate(kind, n, d, int(rng.integers(1, 1000)))
        assert np.array_equal(model(x, depth, B, splits, rng, degenerate), brute(x))
