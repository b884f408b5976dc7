"""Scratch memory of the stateless calls: what a call took beyond 256 MiB is back when it
returns, without anybody's synchronising, and the rest counts as free where a handle
chooses its mode by the free memory."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

KEEP = 256 << 20              # what the library may keep
SLACK = 64 << 20


def _free(km):
    """Free device memory by the driver's count; synchronises nothing."""
    fr, tot = ctypes.c_uint64(0), ctypes.c_uint64(0)
    km.check(km.lib().km_mem_info(0, ctypes.byref(fr), ctypes.byref(tot)), "km_mem_info")
    return fr.value


def _calls(km, X, C, lab):
    return {"assign": lambda: km.assign(X, C, "bf16x3"), "distances": lambda: km.distances(X, C[:2], "bf16x3"),
            "update": lambda: km.update(X, lab, C.shape[0])}


@pytest.mark.parametrize("given_stream", [False, True])
@pytest.mark.parametrize("call", ["assign", "distances", "update"])
def test_memory_is_back_when_a_call_returns(km, gpu, call, given_stream):
    import torch
    with torch.cuda.stream(torch.cuda.Stream() if given_stream else torch.cuda.default_stream()):
        _check_release(km, gpu, call)


def _check_release(km, gpu, call):
    import torch
    # operand copies of 1 GB (assign, distances); a permutation of 800 MB (update)
    n, d = (200000000, 2) if call == "update" else (1000000, 256)
    X = torch.randn(n, d, device=gpu)
    C = torch.randn(64, d, device=gpu)
    lab = torch.randint(0, 64, (n,), dtype=torch.int32, device=gpu)
    small = _calls(km, X[:1000], C, lab[:1000])[call]
    big = _calls(km, X, C, lab)[call]
    big()                                          # torch's own blocks for the outputs are in its cache afterwards
    torch.cuda.synchronize()
    small()
    torch.cuda.synchronize()
    free0 = _free(km)
    big()
    assert free0 - _free(km) <= KEEP + SLACK


def _fill_pool(km, gpu):
    """Leaves between 150 and 256 MiB of scratch with the library."""
    import torch
    X = torch.randn(700000, 64, device=gpu)        # two operand copies of 90 MB
    C = torch.randn(8, 64, device=gpu)
    km.assign(X, C, "bf16x3")
    torch.cuda.synchronize()
    return _free(km)


def test_automatic_panel_choice_counts_kept_memory_as_free(km, gpu):
    free0 = _fill_pool(km, gpu)
    m = km.KernelKMeans(256, 4, 3, panel_rows="auto", precision="fp32")
    free1 = _free(km)
    m.close()
    assert free1 - free0 >= (150 << 20) - SLACK
