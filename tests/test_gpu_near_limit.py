"""The near warps' time limit counts from an error, not from the kernel's start: a join
far longer than the limit returns its count, and one that fails still ends with its
error within it."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture()
def hj():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hilbertjoin_b200 as hj
    L = hj.lib()
    for f in (L.hj_debug_set_near_limit, L.hj_debug_set_wait_gate):
        f.restype, f.argtypes = ctypes.c_int, [ctypes.c_uint64]
    yield hj
    assert L.hj_debug_set_near_limit(0) == 0 and L.hj_debug_set_wait_gate(0) == 0


@pytest.mark.parametrize("form,centring", [("fp16", "global"), ("tf32", "global"), ("bf16x3", "global"),
                                           ("fp16", "block")])
@pytest.mark.parametrize("nbrs", [0.01, 16])  # hardly a near row in the whole join; some in most tiles
def test_a_join_longer_than_the_limit(hj, form, centring, nbrs):
    from hilbertjoin_b200 import workloads as W
    x = W.uniform(250000, 64, 5, dtype=np.float32)
    eps = W.calibrate_eps(x, 250000, nbrs)
    want = hj.self_join_count(x, eps, form="plain")
    assert hj.lib().hj_debug_set_near_limit(1000) == 0  # 1 us
    got, st = hj.self_join_count(x, eps, form=form, centring=centring, return_stats=True)
    assert got == want and st["fp64_items"] == 0 and st["kernel_ms"] > 1.0


def test_an_error_within_the_limit(hj):
    from hilbertjoin_b200 import workloads as W
    x = W.uniform(6000, 32, 3, dtype=np.float32)
    eps = W.calibrate_eps(x, 6000, 16)
    L = hj.lib()
    assert L.hj_debug_set_near_limit(1000) == 0 and L.hj_debug_set_wait_gate(50_000_000) == 0
    with pytest.raises(hj.HJError) as e:
        hj.self_join_count(x, eps, form="fp16")
    assert e.value.status == 4  # HJ_ERR_TIMEOUT
    assert L.hj_debug_set_wait_gate(0) == 0
    assert hj.self_join_count(x, eps, form="fp16") == oracle.self_count_brute(x.astype(np.float64), eps)


def test_limit_longer_than_the_wait_limit_is_rejected(hj):
    assert hj.lib().hj_debug_set_near_limit(3_000_000_000) == 1
