"""Plain form on both sides of the dims where its kernel changes the CTAs per SM or the
dims per B stage: counts and pair lists against the brute-force oracle."""
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


@pytest.mark.parametrize("d", [1, 47, 48, 49, 50, 115, 116, 117, 191, 192, 193, 256])
def test_counts_and_pairs(hj, d):
    x = np.random.default_rng(d).random((1500, d))
    # eps^2 one standard deviation below the mean of |x - y|^2 (d / 6, variance 7 d / 180)
    eps = max(d / 6 - (7 * d / 180) ** 0.5, 1e-4) ** 0.5
    want = O.self_count_brute(x, eps)
    assert want > 0
    assert hj.self_join_count(x, eps, form="plain") == want
    got = hj.self_join_pairs(x, eps, capacity=want)
    dist = ((x[got[:, 0].astype(int)] - x[got[:, 1].astype(int)]) ** 2).sum(1)
    assert len(got) == want and (got[:, 0] < got[:, 1]).all() and dist.max() <= eps * eps * (1 + 1e-12)
