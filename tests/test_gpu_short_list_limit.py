"""The short-list kernels (small.cu) at the longest lists they take and just
past it, against brute force: every arm of the comparison with the other forms
may settle such a list with the same pair loop."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen
from test_gpu_skyline_lists import SHORT, plane, statuses

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [SHORT - 1, SHORT, SHORT + 1])
@pytest.mark.parametrize("kind,d", [("ties", 6), ("anticorrelated", 6), ("plane", 9), ("correlated_q", 16)])
def test_queries(gpu_ctx, kind, d, n):
    """One list of n points; below the limit k_small_skyline takes it whole, and
    with 16 pruners k_small_status what they leave."""
    x = plane(n, d, n) if kind == "plane" else datagen.generate(kind, n, d, 5)
    x[n // 2] = x[0]
    x[n // 3, 0] = -0.0
    full = (1 << d) - 1
    ds = sk.Dataset(gpu_ctx, x)
    for S in (full, full >> 1, full & 0x5555, 0b110, 0b1):
        sky, ext = statuses(x[:, [k for k in range(d) if S >> k & 1]])
        for pq in (0, 16):
            r = sk.skycube(gpu_ctx, ds, subspace=S, pq_size=pq)
            long_list = any(p == "full: pivots+cells" for p, _ in gpu_ctx.last_phases())
            assert long_list == (n > SHORT or pq > 0)
            assert np.array_equal(r.cuboid(S), sky) and np.array_equal(r.extended(S), ext), (S, pq)
            r.close()
    ds.close()


@pytest.mark.parametrize("n", [SHORT - 1, SHORT, SHORT + 1])
def test_per_cuboid_form(gpu_ctx, n):
    """Every point a candidate: the first level's lists have n entries, in one
    k_small_batch launch or through the partition pipeline."""
    d = 5
    x = plane(n, d, n)
    ds = sk.Dataset(gpu_ctx, x)
    r = sk.skycube(gpu_ctx, ds, "sdsc", "plain", want_extended=True)
    assert r.info()["n_candidates"] == n
    for S in (0b11111, 0b01111, 0b10111, 0b11100, 0b00011, 0b00001):
        sky, ext = statuses(x[:, [k for k in range(d) if S >> k & 1]])
        assert np.array_equal(r.cuboid(S), sky) and np.array_equal(r.extended(S), ext), S
    r.close()
    ds.close()
