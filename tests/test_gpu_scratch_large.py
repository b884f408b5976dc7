"""Calls whose scratch goes past what the pool lends (256 MiB) take the rest from cudaMalloc:
several of them at a time, on their own streams and beside small calls, give what each
gives alone, and all of it is back at the end."""
import ctypes
import threading

import pytest

import helpers

pytestmark = pytest.mark.gpu


def test_large_and_small_calls_together(km, gpu):
    import torch
    # candidate lists of 410 and 819 MB, operand copies of 307 MB, a small call
    jobs = []
    for i, (n, d, k, prec) in enumerate([(200000, 16, 300, "bf16"), (400000, 8, 400, "bf16x3"),
                                         (300000, 256, 20, "bf16x3"), (3000, 7, 5, "fp32")]):
        X, _ = helpers.synth_blobs_np(n, d, min(k, 50), -5, 5, 1.0, i)
        jobs.append((torch.from_numpy(X).to(gpu), torch.from_numpy(X[:: n // k][:k].copy()).to(gpu), prec))
    want = [km.assign(*j)[0].clone() for j in jobs]
    torch.cuda.synchronize()
    fr, tot = ctypes.c_uint64(0), ctypes.c_uint64(0)
    km.lib().km_mem_info(0, ctypes.byref(fr), ctypes.byref(tot))
    free0, errors = fr.value, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(8):
                    if not torch.equal(km.assign(*jobs[i])[0], want[i]):
                        errors.append(i)
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not errors, errors
    km.lib().km_mem_info(0, ctypes.byref(fr), ctypes.byref(tot))
    assert free0 - fr.value <= (256 << 20) + (64 << 20)
