"""The preparation kernels at the edges of their tiles and ranges: norm summaries
(padding rows, one and several tiles) through counts that depend on them, and the
dimension cost of dims whose cells fit the shared-memory histogram and of dims
whose cells do not."""
import numpy as np
import pytest

import oracle as O
from hilbertjoin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hj():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hilbertjoin_b200 as hj
    return hj


@pytest.mark.parametrize("n", [1, 31, 33, 255, 256, 257, 2047, 2049, 4100])
def test_norm_summaries_at_tile_edges(hj, n):
    # norms from 1e-6 to 1e2 (d = 64: not folded, every group minimum decides)
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((n, 64)) * np.exp(rng.uniform(-6, 0, (n, 1)))).astype(np.float32)
    x64 = x.astype(np.float64)
    for eps in (0.05, 1.0):
        assert hj.self_join_count(x, eps, form="fp16", centring="global") == O.self_count_brute(x64, eps)


@pytest.mark.parametrize("n", [5, 8192, 20000])
def test_dim_cost_narrow_and_wide_dims(hj, n):
    """Costs against the definition, sum h(h-1)/2 + sum h[c-1] h[c] over the sample's
    cells: dims of 1, 3, 8192, 8193 and 10^6 cells."""
    rng = np.random.default_rng(n)
    x = np.stack([np.zeros(n), *[rng.integers(0, c, n) + 0.5 for c in (3, 8192, 8193, 10**6)]], axis=1)
    if n > 1:
        for j, c in enumerate((3, 8192, 8193, 10**6)):
            x[0, j + 1], x[1, j + 1] = 0.5, c - 0.5  # the whole range occurs
    _, costs = hj.dim_order(x, 1.0, return_costs=True)
    s = min(n, 8192)
    sample = x[(np.arange(s, dtype=np.uint64) * np.uint64(n) // np.uint64(s)).astype(np.int64)]
    for j in range(x.shape[1]):
        cell, h = np.unique(np.floor(sample[:, j]).astype(np.int64), return_counts=True)
        near = sum(int(h[k]) * int(h[k - 1]) for k in range(1, len(cell)) if cell[k] == cell[k - 1] + 1)
        assert int(costs[j]) == int((h.astype(np.int64) * (h - 1) // 2).sum()) + near, j


# the cluster sort's segments (8 CTAs of whole warps, up to 4096 items each), its
# largest size and the first above it; the scatter's own sums (96 tiles of 2048) and
# the first size that scans
@pytest.mark.parametrize("n", [2, 255, 257, 1025, 8192, 8193, 32767, 32768, 32769, 40961, 96 * 2048, 96 * 2048 + 1])
@pytest.mark.parametrize("cells", [2, 50])
def test_ego_order_is_stable_at_the_sort_s_edges(hj, n, cells):
    """perm is the stable order by cell vector: many equal keys (2 cells per dim) and
    several key words (50 cells in 9 dims)."""
    x = np.random.default_rng(n + cells).random((n, 9 if cells > 2 else 3)) * cells
    perm, srt = hj.ego_sort(x, 1.0)
    cell = np.floor(x).astype(np.int64)
    want = np.lexsort([cell[:, t] for t in range(x.shape[1] - 1, -1, -1)])
    assert np.array_equal(perm.astype(np.int64), want)
    assert np.array_equal(srt, x[want])


@pytest.mark.parametrize("form", ["plain", "fp16", "tf32", "bf16x3"])
@pytest.mark.parametrize("active", [0, 3, 5])
@pytest.mark.parametrize("cells", [2, 40, 3000])
def test_counts_with_a_shortened_key(hj, form, active, cells):
    """Keys that end before the last dim (one word at these sizes; more where the
    active dims need them): counts of self-joins, two-set joins, shards and reordered
    dims equal the oracle's, and ref_compat the reference's convention."""
    rng = np.random.default_rng(cells)
    d = 24
    # clusters, so that neighbours exist in every dim's cells
    c = rng.random((12, d)) * cells
    a = (c[rng.integers(0, 12, 1501)] + 0.12 * rng.standard_normal((1501, d))).clip(0, cells)
    b = (c[rng.integers(0, 12, 1203)] + 0.12 * rng.standard_normal((1203, d))).clip(0, cells)
    eps = 0.75
    kw = dict(form=form, active_dims=active)
    want = O.self_count_brute(a, eps)
    assert want > 0
    assert hj.self_join_count(a, eps, **kw) == want
    assert hj.self_join_count(a, eps, reorder_dims=True, **kw) == want
    assert sum(hj.self_join_count(a, eps, shard=(k, 3), **kw) for k in range(3)) == want
    assert hj.join_count(a, b, eps, **kw) == O.join_count_brute(a, b, eps)
    perm, _ = hj.ego_sort(a, eps)
    kept = a[perm[:len(a) // 8 * 8].astype(np.int64)]
    assert hj.self_join_count(a, eps, ref_compat=True, **kw) == O.self_count_brute(kept, eps)


@pytest.mark.parametrize("active", [2, 3, 4])  # 9 and 27 intervals in the warp, 81 by one lane
@pytest.mark.parametrize("kind", ["touching", "gaps"])
def test_stripe_runs_merge(hj, active, kind):
    """Stripe intervals that touch, overlap, repeat and leave gaps, merged into runs:
    the counts equal the oracle's, no tile is visited twice, and none of the load of
    the item sizes changes it (a join of few tiles cuts its items smaller)."""
    rng = np.random.default_rng(active)
    n = 3001
    x = rng.random((n, 6)) * (6.0 if kind == "touching" else 60.0)
    eps = 1.0 if kind == "touching" else 2.0
    want = O.self_count_brute(x, eps)
    for form in ("plain", "fp16"):
        got, st = hj.self_join_count(x, eps, form=form, active_dims=active, return_stats=True)
        assert got == want
        for chunk in (1, 7, 64):
            g2, s2 = hj.self_join_count(x, eps, form=form, active_dims=active, item_chunk=chunk, return_stats=True)
            assert g2 == want and s2["tile_pairs"] == st["tile_pairs"]
    rows = -(-n // 64)
    assert st["tile_pairs"] <= rows * rows


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("d", [2, 5, 33, 64, 65, 128, 129])
def test_index_on_cell_borders(hj, dtype, d):
    # coordinates on, and one ulp beside, the borders of cells of eps: the index takes the
    # neighbour cells from the point's own cell only clear of them. 512-byte rows and
    # longer ones.
    rng = np.random.default_rng(d)
    eps = 0.3
    x = rng.integers(-3, 4, size=(700, d)) * eps * rng.choice([0.0, 0.5, 1.0], size=d, p=[0.6, 0.2, 0.2])
    x[:, 0] = rng.integers(-40, 40, size=700) * eps
    x = x.astype(dtype)
    x = np.where(rng.random(x.shape) < 0.3, np.nextafter(x, dtype(np.inf)), x)
    x = np.where(rng.random(x.shape) < 0.3, np.nextafter(x, dtype(-np.inf)), x).astype(dtype)
    x[350:] = x[:350]
    x[350:, 0] += dtype(eps)  # partners at about eps
    want = O.self_count_brute(x.astype(np.float64), eps)
    assert want > 0
    assert hj.self_join_count(x, eps, form="plain") == want
