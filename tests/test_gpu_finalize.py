"""End of an iteration over its passes of 128 columns and both block sizes (k <= 512 and
above): move, objective and stop against FP64."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 63, 512, 513, 700])
@pytest.mark.parametrize("d", [1, 31, 32, 33, 64, 127, 129, 260])
def test_one_iteration_move_and_objective(km, gpu, k, d):
    n = 3 * k + 40
    X = (np.random.default_rng(k * d).standard_normal((n, d)) * 2).astype(np.float32)
    C0 = X[:k].copy()
    m = km.Lloyd(n, d, k, maxiter=1, init="given").set_data(X)
    lab, cen, r = m.fit(C0=C0)
    m.close()
    it_o, lab_o, cen_o, _ = helpers.orc_lloyd(X, k, 1e-4, 0, 1, C0=C0)
    np.testing.assert_array_equal(lab, lab_o)
    np.testing.assert_array_equal(cen, cen_o)
    move = np.sqrt(((cen.astype(np.float64) - C0) ** 2).sum(1)).max()
    assert abs(r.max_shift - move) <= 1e-12 * move
    obj = ((X.astype(np.float64) - C0[lab]) ** 2).sum()
    # FP32 differences and squares, FP32 partial sums of at most 64 rows
    assert abs(r.objective - obj) <= 70 * 2.0 ** -24 * obj
