"""BF16x3's band is that of its operands, products and FP32 norms alone, at every width:
its column norms are not summed by the tensor cores, whose truncation its fine operands
would show."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hj():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hilbertjoin_b200 as hj
    return hj


@pytest.mark.parametrize("d", [1, 8, 13, 20, 32, 48, 61, 62, 64, 100, 125, 128, 253, 256])
def test_halfwidth(hj, d):
    rng = np.random.default_rng(d)
    a, b = rng.random((700, d)).astype(np.float32), rng.random((900, d)).astype(np.float32)
    _, st = hj.join_count(a, b, 0.3 * d ** 0.5, form="bf16x3", centring="global", return_stats=True)
    terms = 3 * (-(-d // 16) * 16)  # three products per column, 16 columns per MMA step
    want = 1.25 * (3.1 * 2.0 ** -16 + 2 * 2.0 ** -24 + terms * 2.0 ** -22 + 12 * 2.0 ** -24 + d * 2.0 ** -50)
    assert st["band_halfwidth_rel"] == pytest.approx(want, rel=1e-12)
