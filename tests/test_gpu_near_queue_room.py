"""Shapes whose shared memory leaves no near queue: the epilogue classifies every near
row itself. Counts equal the oracle's with hardly any, some and many near rows."""
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


@pytest.mark.parametrize("form,d,centring", [("bf16x3", 192, "global"), ("bf16x3", 193, "global"),
                                             ("bf16x3", 256, "global"), ("tf32", 224, "global"),
                                             ("tf32", 225, "global"), ("tf32", 256, "global"),
                                             ("bf16x3", 61, "block"), ("bf16x3", 62, "block"),
                                             ("bf16x3", 64, "block")])
@pytest.mark.parametrize("nbrs", [0.1, 8, 500])
def test_counts(hj, form, d, centring, nbrs):
    a, b = W.uniform(1213, d, 10 + d, dtype=np.float32), W.uniform(901, d, 11 + d, dtype=np.float32)
    eps = W.calibrate_eps(a, 1213, nbrs)
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    assert hj.self_join_count(a, eps, form=form, centring=centring) == O.self_count_brute(a64, eps)
    assert hj.join_count(a, b, eps, form=form, centring=centring) == O.join_count_brute(a64, b64, eps)


def test_near_rows_hide_behind_the_products(hj):
    """The MMAs of a tile of 256 dims take longer than classifying its near rows: eight
    times the neighbours cost the kernel hardly anything (with a queue of one row per
    warp, which the rows waited for, a fifth)."""
    import torch
    x = W.uniform(60_000, 256, 6, dtype=np.float32)
    ms = {}
    for nbrs in (8, 64):
        eps = W.calibrate_eps(x, 60_000, nbrs)
        dev = torch.from_numpy(x).cuda()
        ms[nbrs] = min(hj.self_join_count(dev, eps, form="bf16x3", return_stats=True)[1]["kernel_ms"]
                       for _ in range(12))
    assert ms[64] < 1.1 * ms[8], ms
