"""A batch's band queue is sized by the tensor-core kernel's work: a job that runs on
the FP64 kernel adds nothing to it, however many candidate pairs it has."""
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu


def test_routed_jobs_add_no_queue():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    code = """
        import torch
        from hilbertjoin_b200.batching import Batch
        n = 400_000
        x = torch.rand(n, 2, device="cuda")
        x[::2] += 1000.0  # two clusters far apart: every item is routed
        used = []
        for eps in (0.001, 0.9):  # few candidate pairs; 4e10
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            with Batch([(x, None, eps)], form="fp16") as b:
                _, st = b.counts(return_stats=True)
                used.append(before - torch.cuda.mem_get_info()[0])
            assert st["fp64_items"] > 0 and st["work_items"] == 0, st
        # (the pool keeps the first batch's buffers: the second figure is what it takes more)
        print(st["candidate_pairs"], *used)
    """
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(code)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    pairs, few, more = map(int, r.stdout.split())
    assert pairs > 3e10
    # work items take 16 bytes per 16 tiles of 64 x 64 pairs, in up to five buffers; a
    # queue for these pairs would be another 16 bytes per 4096 of them
    assert more < 5 * pairs / 4096 + (48 << 20), (few, more)
    assert 16 * pairs / 4096 > 5 * pairs / 4096 + (48 << 20)
