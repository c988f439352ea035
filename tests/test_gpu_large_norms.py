"""Tensor-core forms at coordinates up to their limit (|x| < 1e18), where squared norms
reach 1e36: every real row takes part in the tiles' norm maxima, which the error bound
of a pair stands on, and the counts equal the oracle's."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hj():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hilbertjoin_b200 as hj
    return hj


@pytest.mark.parametrize("form", ["fp16", "tf32", "bf16x3"])
@pytest.mark.parametrize("lo,hi,d,share", [(0.0, 4e14, 2, 0.5), (0.0, 4e15, 1, 0.25), (0.0, 4e15, 1, 0.4),
                                           (-5e16, 5e16, 3, 0.5), (-9e17, 9e17, 2, 0.6), (-9e17, 9e17, 20, 0.9),
                                           (-9e17, 9e17, 64, 0.9), (-9e17, 9e17, 256, 0.95)])
def test_counts(hj, form, lo, hi, d, share):
    rng = np.random.default_rng(d)
    a = rng.uniform(lo, hi, (3000, d)).astype(np.float32)
    b = rng.uniform(lo, hi, (2500, d)).astype(np.float32)
    eps = float(hi - lo) * share * 0.6 * d ** 0.5
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    want = O.join_count_brute(a64, b64, eps)
    assert want > 0
    assert hj.join_count(a, b, eps, form=form, centring="global") == want
    assert hj.self_join_count(a, eps, form=form, centring="global") == O.self_count_brute(a64, eps)
