"""Calls that are given the default stream (NULL) come after the work that is queued
there: inputs still being written by it are read when they are whole, and outputs whose
memory it still uses are written after it.  A long kernel keeps the default stream busy
while the call is made, so a call that does not wait sees the old (valid) values."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

N, D, K = 3000, 24, 7


def _busy():
    import torch
    torch.cuda._sleep(200_000_000)           # about 0.1 s of the default stream


def _data(gpu, seed):
    import torch
    X, _ = helpers.synth_blobs_np(N, D, K, -5, 5, 1.0, seed)
    lab = np.random.default_rng(seed).integers(0, K, N).astype(np.int32)
    return [torch.from_numpy(v).to(gpu) for v in (X, X[:K].copy(), lab)]


def _fit(km, X, **set_data):
    m = km.Lloyd(N, D, K, init="round_robin", maxiter=3, conv="none", precision="bf16")
    getattr(m, set_data.get("call", "set_data"))(X)
    lab, cen, _ = m.fit()
    m.close()
    return lab, cen


def _kernel_fit(km, X):
    m = km.KernelKMeans(N, D, K, kernel="polynomial", gamma=0.01, maxiter=3, precision="fp32").set_data(X)
    lab, _ = m.fit()
    m.close()
    return (lab,)


CALLS = {
    "assign": lambda km, X, C, lab: km.assign(X, C, "bf16x3", want_mindist=True)[:2],
    "assign_fp32": lambda km, X, C, lab: km.assign(X, C, "fp32")[:1],
    "distances": lambda km, X, C, lab: (km.distances(X, C, "fp32"),),
    "update": lambda km, X, C, lab: km.update(X, lab, K),
    "kernel_matrix": lambda km, X, C, lab: (km.kernel_matrix(X, "gaussian", sigma=3.0, precision="bf16x3"),),
    "lloyd_set_data": lambda km, X, C, lab: _fit(km, X),
    "lloyd_set_data_bf16": lambda km, X, C, lab: _fit(km, X.view(-1).to(dtype=_bf16()), call="set_data_bf16"),
    "kkm_set_data": lambda km, X, C, lab: _kernel_fit(km, X),
}


def _bf16():
    import torch
    return torch.bfloat16


def _host(out):
    return [o if isinstance(o, np.ndarray) else o.cpu().numpy() for o in out]


@pytest.mark.parametrize("call", sorted(CALLS))
def test_inputs_written_on_the_default_stream(km, gpu, call):
    import torch
    old, new = _data(gpu, 1), _data(gpu, 2)
    torch.cuda.synchronize()
    want = _host(CALLS[call](km, *new))                  # (also loads and warms everything up)
    stale = _host(CALLS[call](km, *old))
    assert any(not np.array_equal(a, b) for a, b in zip(want, stale))
    bufs = [t.clone() for t in old]
    torch.cuda.synchronize()
    _busy()
    for b, t in zip(bufs, new):
        b.copy_(t)
    got = CALLS[call](km, *bufs)
    for a, b in zip(want, _host(got)):
        np.testing.assert_array_equal(b, a)


def test_outputs_in_memory_that_the_default_stream_still_uses(km, gpu):
    import torch
    X, C, _ = _data(gpu, 3)
    want = km.assign(X, C, "bf16")[0].cpu().numpy()
    torch.empty(N, dtype=torch.int32, device=gpu).fill_(-1)   # (the fill's kernel is loaded)
    torch.cuda.synchronize()
    before = torch.empty(N, dtype=torch.int32, device=gpu)
    at = before.data_ptr()
    _busy()
    before.fill_(-1)                                     # queued behind the long kernel
    del before                                           # the caching allocator hands the block out again
    lab = km.assign(X, C, "bf16")[0]
    assert lab.data_ptr() == at
    torch.cuda.synchronize()
    np.testing.assert_array_equal(lab.cpu().numpy(), want)


def test_inputs_written_on_a_blocking_stream(km, gpu):
    """The default stream follows every blocking stream, so a call without a stream does."""
    import ctypes
    import torch
    lib = [line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line]
    if not lib:
        pytest.skip("no shared CUDA runtime in this process")
    rt, raw = ctypes.CDLL(lib[0]), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(raw)) == 0
    old, new = _data(gpu, 5), _data(gpu, 6)
    want = _host(CALLS["assign"](km, *new))
    bufs = [t.clone() for t in old]
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.ExternalStream(raw.value)):
        _busy()
        for b, t in zip(bufs, new):
            b.copy_(t)
    got = _host(CALLS["assign"](km, *bufs))
    torch.cuda.synchronize()
    rt.cudaStreamDestroy(raw)
    for a, b in zip(want, got):
        np.testing.assert_array_equal(b, a)
