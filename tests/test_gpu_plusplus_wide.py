"""Seeded k-means++ of rows of more than 256 columns (32 rows a warp and step, chunks of 1024
rows), at the edges of both: picked rows equal to the oracle's."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(31, 257, 3), (32, 259, 32), (33, 300, 7), (255, 512, 5), (1023, 288, 20), (1024, 784, 6),
                                   (1057, 400, 60), (2081, 513, 9)])
def test_wide_rows_match_the_oracle(km, gpu, n, d, k):
    X, _ = helpers.synth_blobs_np(n, d, max(2, k // 3), -4, 4, 1.5, 7 * d + k)
    m = km.Lloyd(n, d, k, seed=11, init="plusplus", maxiter=1).set_data(X)
    C = m.init_centroids()
    m.close()
    np.testing.assert_array_equal(C, X[helpers.orc_plusplus(X, k, 11)])
