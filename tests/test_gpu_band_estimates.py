"""max_abs_err_band is the largest |est - dist2| over the band pairs, also where most of
a group's rows are near (with block centres it may leave those out). Bounds on it from the estimates of every pair (the same
operands, so the same values): a pair whose estimate and exact distance lie on
different sides of eps^2 is certainly in the band, and no band pair is off by more than
the worst of all pairs."""
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


@pytest.mark.parametrize("form", ["fp16", "tf32", "bf16x3"])
@pytest.mark.parametrize("centring", ["global", "block"])
@pytest.mark.parametrize("d", [20, 32, 64])  # folded norms, norms outside (TF32), norms outside
@pytest.mark.parametrize("q", [0.02, 0.5])  # few near rows per group, and nearly all
def test_statistic_covers_the_band(hj, form, centring, d, q):
    rng = np.random.default_rng(100 * d)
    a, b = rng.random((2100, d)).astype(np.float32), rng.random((1900, d)).astype(np.float32)
    exact = ((a[:, None, :].astype(np.float64) - b[None, :, :]) ** 2).sum(-1)
    eps = float(np.sqrt(np.quantile(exact, q)))
    est, st = hj.tc_estimates(a, b, form, centring=centring, eps=eps, return_stats=True)
    _, st = hj.join_count(a, b, eps, form=form, centring=centring, active_dims=0, return_stats=True)
    assert st["fp64_items"] == 0 and st["band_pairs"] > 0
    seen = np.isfinite(est)  # pairs of the work list
    err = np.where(seen, np.abs(est.astype(np.float64) - exact), 0.0)
    crossed = seen & ((est <= eps * eps) != (exact <= eps * eps))
    assert crossed.any()
    # the statistic is the FP32 rounding of one pair's error
    assert st["max_abs_err_band"] <= err.max() * (1 + 2.0 ** -23)
    if centring == "global":
        assert st["max_abs_err_band"] >= err[crossed].max() * (1 - 2.0 ** -23) > 0


@pytest.mark.parametrize("form", ["fp16", "tf32", "bf16x3"])
def test_statistic_of_a_batch(hj, form):
    """A batch of the same joins: the largest of the jobs' own statistics."""
    import torch
    from hilbertjoin_b200.batching import Batch
    rng = np.random.default_rng(9)
    jobs, worst = [], 0.0
    for d in (20, 64):
        x = rng.random((1500, d)).astype(np.float32)
        eps = float(np.sqrt(np.median(((x[:300, None].astype(np.float64) - x[None, 300:600]) ** 2).sum(-1))))
        _, st = hj.self_join_count(x, eps, form=form, centring="global", return_stats=True)
        worst = max(worst, st["max_abs_err_band"])
        jobs.append((torch.from_numpy(x).cuda(), None, eps))
    assert worst > 0
    b = Batch(jobs, form=form)
    _, st = b.counts(return_stats=True)
    assert st["max_abs_err_band"] == worst
