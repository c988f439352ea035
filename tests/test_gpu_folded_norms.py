"""Tensor-core joins whose column norms are folded into the MMA (three operand
columns that fit the last 128-byte atom) and those whose norms stay outside:
counts equal the oracle's at the edges of the column budget, with many near rows
in a group (the epilogue's own classification), with few (the near queues), in
self-joins (the triangle mask), ragged sizes and padding rows."""
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


# FP16 and BF16x3 atoms hold 64 columns, TF32 atoms 32: the last folded width, the
# first that is not, and a multi-atom one
@pytest.mark.parametrize("form", ["fp16", "tf32", "bf16x3"])
@pytest.mark.parametrize("d", [1, 13, 29, 30, 61, 62, 64, 125, 126, 253, 256])
@pytest.mark.parametrize("nbrs", [2, 300])
def test_counts_at_the_column_budget(hj, form, d, nbrs):
    a, b = W.uniform(1213, d, 10 + d, dtype=np.float32), W.uniform(901, d, 11 + d, dtype=np.float32)
    eps = W.calibrate_eps(a, 1213, nbrs)
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    assert hj.self_join_count(a, eps, form=form, centring="global") == O.self_count_brute(a64, eps)
    assert hj.join_count(a, b, eps, form=form, centring="global") == O.join_count_brute(a64, b64, eps)


@pytest.mark.parametrize("form", ["fp16", "bf16x3"])
def test_norms_that_differ_within_a_group(hj, form):
    """Many occupied cells and norms over four decades: 32 consecutive ranks differ
    widely in norm, so only the folded accumulator orders a row's columns."""
    rng = np.random.default_rng(5)
    x = (rng.standard_normal((5000, 20)) * np.exp(rng.uniform(-4.5, 0, (5000, 1)))).astype(np.float32)
    x64 = x.astype(np.float64)
    for q in (0.002, 0.2):
        d2 = ((x64[:300, None] - x64[None, 300:600]) ** 2).sum(-1)
        eps = float(np.sqrt(np.quantile(d2, q)))
        assert hj.self_join_count(x, eps, form=form, centring="global") == O.self_count_brute(x64, eps)
