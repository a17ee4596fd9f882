"""Branches that only large inputs or many pruners reach: a prefilter whose
tables need a second launch (prefilter.cu), the compaction of more than 4,096
status blocks (prep.cu, status_write) and the scan of more than 4,096 blocks of
counts (launch_scan_counts)."""
import numpy as np
import pytest

import skycube_gb300 as sk
from skycube_gb300 import datagen
from test_gpu_skyline_lists import statuses

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,pq", [(16, 769), (16, 1000), (16, 1024), (15, 1024), (14, 897), (13, 1024)])
@pytest.mark.parametrize("kind", ["ties", "uniform", "correlated_q"])
def test_pruner_tables_in_two_launches(gpu_ctx, kind, d, pq):
    """More than 200 KB of tables: K > 768 at 16 attributes, 832, 896 and 960
    at 15, 14 and 13."""
    x = datagen.generate(kind, 7000, d, d + pq)
    full = (1 << d) - 1
    ds = sk.Dataset(gpu_ctx, x)
    for S in (full, full & 0x5b5b):
        sky, ext = statuses(x[:, [k for k in range(d) if S >> k & 1]])
        r = sk.skycube(gpu_ctx, ds, subspace=S, pq_size=pq)
        assert any(p == "full: prefilter" for p, _ in gpu_ctx.last_phases())
        assert np.array_equal(r.cuboid(S), sky) and np.array_equal(r.extended(S), ext), S
        r.close()
    ds.close()


@pytest.mark.parametrize("pq_size", [0, -1])
def test_compaction_of_many_blocks(gpu_ctx, pq_size):
    """4,300,001 points: 40,000 of the line y = -x, no two comparable, at random
    places, 1,000 copies of some of them with one attribute raised (dominated,
    not strictly), the rest strictly dominated by the line's middle."""
    n, line, raised = 4300001, 40000, 1000
    rng = np.random.default_rng(3)
    u = rng.permutation(np.arange(1, line + 1)).astype(np.float32)
    x = (line + rng.random((n, 2)) * 1000).astype(np.float32)
    at = rng.permutation(n)[:line + raised]
    x[at[:line], 0] = u
    x[at[:line], 1] = -u
    x[at[line:], 0] = u[:raised] + np.float32(0.5)
    x[at[line:], 1] = -u[:raised]
    ds = sk.Dataset(gpu_ctx, x)
    r = sk.skycube(gpu_ctx, ds, subspace=3, pq_size=pq_size)
    assert np.array_equal(r.cuboid(3), np.sort(at[:line]))
    assert np.array_equal(r.extended(3), np.sort(at[line:]))
    r.close()
    ds.close()


def test_scan_of_many_count_blocks(gpu_ctx):
    """16 attributes and 530,000 candidates: 65,536 columns by 259 row tiles,
    16.97 M counts, against the level form's lists."""
    n, d = 530000, 16
    x = np.random.default_rng(9).random((n, d), dtype=np.float32)
    x[:, 0] = d - x[:, 1:].sum(axis=1)
    ds = sk.Dataset(gpu_ctx, x)
    a = sk.skycube(gpu_ctx, ds, max_d=2, form="bitmaps")
    b = sk.skycube(gpu_ctx, ds, max_d=2, form="levels")
    assert a.form()[0] == "bitmaps" and b.form()[0] == "levels"
    assert a.info() == b.info() and a.info()["n_candidates"] > 256 * 2048 + 1
    for c in [c for c in range(1, 1 << d) if bin(c).count("1") <= 2] + [(1 << d) - 1]:
        assert np.array_equal(a.cuboid(c), b.cuboid(c)), c
    for o in (a, b, ds):
        o.close()
