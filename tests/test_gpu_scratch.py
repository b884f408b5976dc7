"""The scratch pool of the stateless calls: results do not depend on other
threads and streams that use it at the same time, and what it keeps between
calls is bounded (256 MiB)."""
import threading

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def test_scratch_is_safe_across_threads_and_streams(km, gpu):
    import torch
    jobs = []
    for i, (n, d, k) in enumerate([(5000, 16, 20), (70001, 33, 64), (20000, 128, 200), (900, 7, 3)]):
        X, _ = helpers.synth_blobs_np(n, d, k, -5, 5, 1.0, i)
        C = X[:: n // k][:k].copy()
        jobs.append((torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), k))
    torch.cuda.synchronize()
    want = []
    for X, C, k in jobs:
        lab = km.assign(X, C, "bf16x3")[0]
        want.append((lab.clone(), km.update(X, lab, k)[0].clone()))
    errors = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                X, C, k = jobs[i]
                for _ in range(25):
                    lab = km.assign(X, C, "bf16x3")[0]
                    cen = km.update(X, lab, k)[0]
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(lab, want[i][0]) or not torch.equal(cen, want[i][1]):
                        errors.append(i)
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors


def test_scratch_kept_between_calls_is_bounded(km, gpu):
    import torch
    X = torch.randn(1000000, 256, device=gpu)
    C = torch.randn(64, 256, device=gpu)
    km.assign(X[:1000], C, "bf16x3")
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    km.assign(X, C, "bf16x3")              # over 1 GB of operand copies
    torch.cuda.synchronize()
    km.assign(X[:1000], C, "bf16x3")
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] <= (256 << 20) + (64 << 20)
    assert np.isfinite(C.sum().item())
