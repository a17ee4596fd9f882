"""Short lists (small.cu, k_small_skyline): one launch that compares all pairs
and compacts in the last CTA, against brute-force statuses, as a subspace
query, a skycube and the per-cuboid form, around its edges (groups of 32
points, tiles of 512 and 1,024 q's, the longest list it takes and one more)."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen
from test_gpu_skyline_tree import brute

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 511, 513, 1023, 1025, 2047])
@pytest.mark.parametrize("kind,d", [("uniform", 2), ("ties", 5), ("anticorrelated", 9),
                                    ("correlated_q", 16)])
def test_queries(gpu_ctx, n, kind, d):
    x = datagen.generate(kind, n, d, 31 * n + d)
    if n > 4:
        x[n // 2] = x[0]      # an equal point
        x[n // 3, 0] = -0.0   # a signed zero
    ds = sk.Dataset(gpu_ctx, x)
    full = (1 << d) - 1
    for S in (full, full & 0b1010101010101010, 1):
        if not S:
            continue
        sky, ext = brute(x[:, [k for k in range(d) if S >> k & 1]])
        r = sk.skycube(gpu_ctx, ds, subspace=S)
        assert np.array_equal(r.cuboid(S), sky) and np.array_equal(r.extended(S), ext), (n, S)
        info = r.info()
        fsky, fext = brute(x)
        assert info["n_candidates"] == len(fsky) + len(fext)
        assert info["total_skyline_ids"] == len(sky)
        r.close()
    ds.close()


@pytest.mark.parametrize("kind,d", [("ties", 6), ("anticorrelated", 6)])
@pytest.mark.parametrize("n", [6143, 6144, 6145])
def test_longest_list_and_the_pipeline_agree(gpu_ctx, kind, d, n):
    x = datagen.generate(kind, n, d, 5)
    ds = sk.Dataset(gpu_ctx, x)
    a = sk.skycube(gpu_ctx, ds, want_extended=True)
    b = sk.skycube(gpu_ctx, ds, want_extended=True, pq_size=16)  # the pipeline
    c = sk.skycube(gpu_ctx, ds, "sdsc", "plain", want_extended=True)
    for S in range(1, 1 << d):
        for o in (b, c):
            assert np.array_equal(a.cuboid(S), o.cuboid(S)), S
            assert np.array_equal(a.extended(S), o.extended(S)), S
    for o in (a, b, c, ds):
        o.close()


@pytest.mark.parametrize("kind,n,d,max_d", [
    ("uniform", 33, 4, 0), ("ties", 3000, 9, 0), ("anticorrelated", 1500, 9, 0),
    ("anticorrelated", 30000, 6, 0), ("correlated_q", 40000, 10, 3), ("uniform", 60000, 8, 5),
])
def test_levels_of_the_per_cuboid_form(gpu_ctx, kind, n, d, max_d):
    """k_small_batch: a lattice level's short lists in one launch, more than 64
    of them in several (9 attributes: 126 on two levels), beside longer lists
    of the same level, with parents from either, against the bitmap form."""
    ds = sk.Dataset(gpu_ctx, datagen.generate(kind, n, d, 3 * n + d))
    a = sk.skycube(gpu_ctx, ds, max_d=max_d, want_extended=True, form="bitmaps")
    b = sk.skycube(gpu_ctx, ds, "sdsc", "plain", max_d=max_d, want_extended=True)
    top = max_d or d
    for S in range(1, 1 << d):
        if bin(S).count("1") <= top or S == (1 << d) - 1:
            assert np.array_equal(a.cuboid(S), b.cuboid(S)), S
            assert np.array_equal(a.extended(S), b.extended(S)), S
    for o in (a, b, ds):
        o.close()


@pytest.mark.parametrize("open_points", [1, 33, 2049, 4095, 4096, 4097, 6143, 6144, 6145])
@pytest.mark.parametrize("d", [3, 8, 13])
def test_few_points_left_by_the_prefilter(gpu_ctx, open_points, d):
    """k_small_status and the emptied pipeline, around the longest list it
    takes: `open_points` points of a plane, a tenth of them repeated with one
    attribute raised (dominated, not strictly), and 40,000 points that all of
    them strictly dominate; then with three equal points below everything."""
    rng = np.random.default_rng(open_points + d)
    e = rng.exponential(size=(open_points, d))
    a = (e / e.sum(axis=1, keepdims=True)).astype(np.float32)
    t = open_points // 10
    if t:
        a[-t:] = a[:t]
        a[-t:, rng.integers(0, d, t)] += np.float32(0.125)
    x = np.concatenate([a, (2 + rng.random((40000, d))).astype(np.float32)])
    at = rng.permutation(len(x))
    x = np.ascontiguousarray(x[at])
    back = np.flatnonzero(at < open_points)  # where the plane's points went
    sky, ext = brute(x[back])
    sky, ext = back[sky], back[ext]
    ds = sk.Dataset(gpu_ctx, x)
    full = (1 << d) - 1
    for pq in (0, 64, 512):
        r = sk.skycube(gpu_ctx, ds, subspace=full, pq_size=pq)
        assert np.array_equal(r.cuboid(full), sky) and np.array_equal(r.extended(full), ext), pq
        r.close()
    ds.close()
    x[7] = x[4099] = x[30000] = -1.0
    ds = sk.Dataset(gpu_ctx, x)
    r = sk.skycube(gpu_ctx, ds, subspace=full)
    assert np.array_equal(r.cuboid(full), [7, 4099, 30000]) and len(r.extended(full)) == 0
    r.close()
    ds.close()
