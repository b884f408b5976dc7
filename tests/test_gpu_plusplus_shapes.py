"""Seeded k-means++ at the edges of the cost kernels' tiles (256 rows, 128 above
d = 128, a warp per row above d = 256), of the candidate counts (4, 8, 16 a
thread) and of the sampler's chunks: picked rows equal to the oracle's."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(5, 1, 5), (255, 2, 7), (256, 3, 8), (257, 31, 9), (1023, 32, 20), (1024, 33, 21),
                                   (1025, 64, 60), (3000, 127, 150), (2049, 128, 12), (700, 129, 30), (900, 255, 9),
                                   (1500, 256, 25), (1500, 257, 25), (2500, 300, 8), (9000, 5, 450), (40000, 7, 3)])
def test_plusplus_picks_match_the_oracle(km, gpu, n, d, k):
    X, _ = helpers.synth_blobs_np(n, d, max(2, k // 3), -4, 4, 1.5, 31 * d + k)
    m = km.Lloyd(n, d, k, seed=5, init="plusplus", maxiter=1).set_data(X)
    C = m.init_centroids()
    m.close()
    np.testing.assert_array_equal(C, X[helpers.orc_plusplus(X, k, 5)])


def test_plusplus_costs_beyond_the_fp32_range(km, gpu):
    """Distances near 1e37: a tile's cost passes the FP32 range, the FP64 total does not."""
    X, _ = helpers.synth_blobs_np(1000, 4, 5, -4, 4, 1.0, 3)
    X = (X * np.float32(3e17)).astype(np.float32)
    m = km.Lloyd(1000, 4, 12, seed=5, init="plusplus", maxiter=1).set_data(X)
    C = m.init_centroids()
    m.close()
    np.testing.assert_array_equal(C, X[helpers.orc_plusplus(X, 12, 5)])
