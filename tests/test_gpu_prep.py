"""Point preparation (norms, copy, BF16 operands) over the groups of lanes a row is given:
columns at the edges of a step, row counts at the edges of a round, inputs that are and are
not 16-byte aligned.  Fits equal the CPU oracle's label for label and centroid for centroid,
also when the caller's buffer is overwritten once the points are set."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

SHAPES = [(7, 1), (40, 3), (33, 4), (130, 8), (129, 9), (50, 14), (70, 16), (65, 20), (257, 36), (75, 50), (64, 64), (61, 68), (300, 100),
          (131, 128), (44, 126), (50, 130), (66, 129), (45, 132), (90, 516), (35, 601)]


@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("precision", ["fp32", "bf16x3", "bf16"])
@pytest.mark.parametrize("n,d", SHAPES)
def test_prep_fit_vs_oracle(km, gpu, n, d, precision, shift):
    import torch
    Xh = helpers.synth_blobs_np(n, d, 3, -1, 1, 0.4, n + d)[0].astype(np.float32)
    buf = torch.zeros(n * d + 4, device=gpu)
    X = buf[shift: shift + n * d].view(n, d)     # rows start 16, 4 or 8 bytes aligned
    X.copy_(torch.from_numpy(Xh))
    it_o, lab_o, cen_o, _ = helpers.orc_lloyd(Xh, 3, 1e-4, 1, 6)
    m = km.Lloyd(n, d, 3, tol=1e-4, seed=1, maxiter=6, precision=precision).set_data(X)
    X.zero_()
    lab, cen, r = m.fit()
    m.close()
    np.testing.assert_array_equal(lab, lab_o)
    np.testing.assert_array_equal(cen, cen_o)


@pytest.mark.parametrize("n,d", [(40, 3), (130, 8), (70, 64), (61, 128), (45, 132)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_prep_rejects_nonfinite(km, gpu, n, d, bad):
    X = helpers.synth_blobs_np(n, d, 3, -1, 1, 0.4, 1)[0].astype(np.float32)
    m = km.Lloyd(n, d, 3, maxiter=2)
    for at in ((0, 0), (n - 1, d - 1), (n // 2, d // 2)):
        Y = X.copy()
        Y[at] = bad
        with pytest.raises(km.KmError) as e:
            m.set_data(Y)
        assert e.value.status == km.KM_ERR_ARG
    m.close()
