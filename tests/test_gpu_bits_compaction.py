"""The compaction of bitmaps into per-cuboid id lists (mdmc.cu, k_bits_count
and k_bits_write) against the per-point bitmaps themselves: candidate counts
around the edges of its 32-row groups, its tiles (64 rows and more) and staged 128-row steps,
one word per row up to 1,024, sparse and dense columns, skylines and extended
skylines, and caps (words with no wanted column)."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen

pytestmark = pytest.mark.gpu


def on_a_plane(n, d, seed):
    """n points none of which dominates another on the full space."""
    x = np.random.default_rng(seed).integers(0, 1 << 10, size=(n, d)).astype(np.float32)
    x[:, 0] = (1 << 14) - x[:, 1:].sum(axis=1)
    return x


def check_lists(r, d, max_d, n):
    bits, pids = r.bitmaps()
    assert np.array_equal(pids, np.arange(n))  # every point is a candidate
    total = 0
    for c in range(1, 1 << d):
        dominated = (bits[:, c >> 5] >> np.uint32(c & 31)) & 1
        want = pids[dominated == 0]
        assert np.array_equal(r.cuboid(c), want), (n, d, c)
        total += len(want)
    assert r.info()["total_skyline_ids"] == total


@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 255, 257, 1000, 2049])
@pytest.mark.parametrize("d", [2, 4, 6, 9])
def test_lists_equal_the_bitmaps(gpu_ctx, n, d):
    ds = sk.Dataset(gpu_ctx, on_a_plane(n, d, 10 * n + d))
    r = sk.skycube(gpu_ctx, ds, want_bitmaps=True)
    check_lists(r, d, d, n)
    r.close()
    ds.close()


@pytest.mark.parametrize("d,max_d", [(11, 2), (13, 3), (15, 5), (11, 11)])
def test_wide_rows_and_caps(gpu_ctx, d, max_d):
    x = datagen.generate("ties", 3001, d, d)
    ds = sk.Dataset(gpu_ctx, x)
    a = sk.skycube(gpu_ctx, ds, max_d=max_d, want_extended=True, form="bitmaps")
    b = sk.skycube(gpu_ctx, ds, want_bitmaps=True, want_extended=True)
    bits, pids = b.bitmaps()
    full = (1 << d) - 1
    for c in range(1, full + 1):
        if bin(c).count("1") > max_d and c != full:
            assert len(a.cuboid(c)) == 0 and len(a.extended(c)) == 0
            continue
        dominated = (bits[:, c >> 5] >> np.uint32(c & 31)) & 1
        assert np.array_equal(a.cuboid(c), pids[dominated == 0]), (d, c)
        assert np.array_equal(a.extended(c), b.extended(c)), (d, c)
    for o in (a, b, ds):
        o.close()
