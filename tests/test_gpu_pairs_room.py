"""Pair lists whose length meets the caller's capacity and the listing run's first
buffer (2^23 pairs): exactly full, one short, number only, and a second run."""
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


@pytest.mark.parametrize("n,d", [(65, 3), (700, 5), (1111, 17)])
def test_capacity_edges(hj, n, d):
    x = np.random.default_rng(n).random((n, d))
    eps = 0.25 * d ** 0.5  # some pairs at every d (the oracle counts them)
    total = O.self_count_brute(x, eps)
    assert total > 2
    got = hj.self_join_pairs(x, eps, capacity=total)
    dist = ((x[got[:, 0].astype(int)] - x[got[:, 1].astype(int)]) ** 2).sum(1)
    assert len(got) == total and (got[:, 0] < got[:, 1]).all() and dist.max() <= eps * eps * (1 + 1e-12)
    key = got[:, 0].astype(np.int64) * n + got[:, 1].astype(np.int64)
    assert (np.diff(key) > 0).all()  # sorted, each pair once
    for cap in (total - 1, 0):
        with pytest.raises(hj.HJError) as e:
            hj.self_join_pairs(x, eps, capacity=cap)
        assert e.value.status == hj.ERR_CAPACITY


def test_more_pairs_than_the_first_buffer(hj):
    n = 4200  # every pair: 8,817,900 > 2^23
    x = np.random.default_rng(1).random((n, 2))
    got = hj.self_join_pairs(x, 10.0)
    want = np.stack(np.triu_indices(n, 1), axis=1)
    assert np.array_equal(got.astype(np.int64), want)
