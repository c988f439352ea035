"""The work list of a self-join holds each tile pair once: in every form at most the
tile pairs on or above the diagonal, fewer where the stripes leave gaps, and the same
number however the items are cut."""
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


@pytest.mark.parametrize("active", [1, 2, 3, 4, 5])  # 3 to 27 intervals in the warp, 81 and 243 by one lane
@pytest.mark.parametrize("kind", ["touching", "gaps"])
@pytest.mark.parametrize("form,tile_a,tile_b", [("plain", 64, 64), ("fp16", 128, 256)])
def test_tile_pairs(hj, active, kind, form, tile_a, tile_b):
    n = 3001
    x = np.random.default_rng(active).random((n, 6)) * (6.0 if kind == "touching" else 60.0)
    eps = 1.0 if kind == "touching" else 2.0
    ta, tb = -(-n // tile_a), -(-n // tile_b)
    upper = sum(tb - i * tile_a // tile_b for i in range(ta))
    got, st = hj.self_join_count(x, eps, form=form, active_dims=active, return_stats=True)
    assert got == O.self_count_brute(x, eps)
    # every tile meets itself; with gaps (30 cells in the first dim, 3 of which matter) most
    # of the rest drop out
    assert ta <= st["tile_pairs"] <= upper
    if kind == "gaps":
        assert st["tile_pairs"] < 0.6 * upper
    for chunk in (1, 7, 64):
        _, s2 = hj.self_join_count(x, eps, form=form, active_dims=active, item_chunk=chunk, return_stats=True)
        assert s2["tile_pairs"] == st["tile_pairs"]
