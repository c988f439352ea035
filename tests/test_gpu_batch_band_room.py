"""Every run of a planned batch fits its band queue: the slots that warps reserve and
leave unused differ from run to run, so a queue that the planning run just filled may
not hold the next one's."""
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


def test_runs_near_the_queue_s_size(hj):
    import torch
    from hilbertjoin_b200.batching import Batch
    g = torch.Generator(device="cuda").manual_seed(3)
    d = 32
    a = torch.rand(60000, d, generator=g, device="cuda")
    c = torch.rand(1900, d, generator=g, device="cuda")
    # partners in clumps of 32: a near row has up to 32 band pairs, and the near warps, who
    # reserve for as many rows as are queued at the time, take other slots in every run
    b = (c.repeat_interleave(32, 0) + 2e-4 * torch.rand(1900 * 32, d, generator=g, device="cuda")).contiguous()
    dist = torch.cdist(a[:2000].double(), c[:1000].double()).flatten()

    def band(eps):
        return hj.join_count(a, b, eps, form="fp16", return_stats=True)[1]["band_pairs"]

    # the queue of a small batch: 2^20 pairs, and 32 slots for each of 10 warps per SM
    slack = hj.lib().hj_device_sm_count(-1) * 10 * 32
    cap = (1 << 20) + slack
    lo, hi = (float(torch.quantile(dist, q)) for q in (0.001, 0.02))
    assert band(lo) < (1 << 20) and band(hi) > cap
    # of the slots that the warps may leave unused, 35 to 45% are, as a rule
    for back in range(int(0.45 * slack), int(0.35 * slack), -40):
        while hi - lo > 1e-7 * hi:
            mid = 0.5 * (lo + hi)
            lo, hi = (mid, hi) if band(mid) < cap - back else (lo, mid)
        want = hj.join_count(a, b, lo, form="fp16")
        with Batch([(a, b, lo)], form="fp16") as batch:
            for _ in range(8):
                batch.run()
                assert batch.counts() == [want]
        hi = lo * 1.001
    assert want == hj.join_count(a, b, lo, form="plain")
