"""set_data of points in memory that is not the device's own: they are copied, not read in
place (managed memory here; another GPU's memory takes the same way)."""
import ctypes

import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def _runtime():
    """The CUDA runtime that torch has loaded."""
    for line in open("/proc/self/maps"):
        if "libcudart" in line:
            return ctypes.CDLL(line.split()[-1])
    pytest.skip("no shared CUDA runtime in this process")


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
@pytest.mark.parametrize("d", [5, 16])
def test_points_in_managed_memory(km, gpu, precision, d):
    rt = _runtime()
    n, k = 3000, 6
    X, _ = helpers.synth_blobs_np(n, d, k, -5, 5, 1.0, 4)
    p = ctypes.c_void_p()
    assert rt.cudaMallocManaged(ctypes.byref(p), ctypes.c_size_t(X.nbytes), ctypes.c_uint(1)) == 0
    try:
        ctypes.memmove(p.value, X.ctypes.data, X.nbytes)
        m = km.Lloyd(n, d, k, seed=2, maxiter=8, precision=precision)
        km.check(km.lib().km_lloyd_set_data(m.h, p.value, 1), "km_lloyd_set_data")
        ctypes.memset(p.value, 0, X.nbytes)              # the handle keeps its own copy
        lab, cen, r = m.fit()
        m.close()
    finally:
        rt.cudaFree(p)
    it_o, lab_o, cen_o, _ = helpers.orc_lloyd(X, k, 1e-4, 2, 8)
    assert r.converged_iter == it_o
    np.testing.assert_array_equal(lab, lab_o)
    np.testing.assert_array_equal(cen.view(np.uint32), cen_o.view(np.uint32))
