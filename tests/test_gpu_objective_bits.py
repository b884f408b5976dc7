"""The objective of rows that are not 16-byte aligned is summed as if in FP64.  One cluster at
the origin and whole-numbered points: every row's distance, and every sum of 16 of one
coordinate, is exact in FP32, and the whole sum needs 53 bits or fewer, but its parts lie
so far apart (2^47, runs of 2^22 that pile up below the first part's last bit, single ones)
that a sum held in two FP32 parts loses the ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 5, 6, 7])
def test_objective_of_parts_far_apart(km, gpu, d):
    big, mid, ones = 128, 128 * 16, 128 * 40          # rows: whole batches of the sums
    x = np.zeros(big + mid + ones, np.float32)
    x[:big] = 2.0 ** 21                               # squares 2^42: 32 rows of a lane make 2^47
    x[big:big + mid] = 2.0 ** 9                       # squares 2^18: runs of 16 make 2^22
    x[big + mid::128] = 1.0                           # one row of each further batch
    X = np.ascontiguousarray(np.repeat(x[:, None], d, axis=1))
    want = d * int((x.astype(np.float64) ** 2).sum())
    assert want < 2 ** 53
    m = km.Lloyd(len(x), d, 1, init="given", maxiter=1, conv="none", precision="fp32").set_data(X)
    _, _, r = m.fit(np.zeros((1, d), np.float32))
    m.close()
    assert int(r.objective) == want and r.objective == float(want)
