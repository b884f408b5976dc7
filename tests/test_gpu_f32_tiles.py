"""FP32 distance kernel at the edges of its tiles (32, 48, 64, 96, 128 centroids
and chunks of them; 64, 128 or 256 rows), of its coordinate stages and of the
candidate lists (groups of 1..12 equal centroids: single candidates, short
queue, full re-score): labels equal to the oracle's for every row."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 31, 32, 33, 48, 49, 64, 65, 96, 97, 128, 129, 192, 193, 257, 400])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 191, 193, 257, 1000])
def test_f32_labels_at_tile_edges(km, gpu, n, k):
    import torch
    if k > n:
        pytest.skip("k > n")
    d = (1, 3, 7, 8, 16, 17, 20, 36, 50)[(n + k) % 9]
    rng = np.random.default_rng(1000 * n + k)
    X = (rng.standard_normal((n, d)) * 3).astype(np.float32)
    C = X[rng.choice(n, k, replace=False)].copy()
    for g in range(1, min(12, k // 4)):                    # groups of equal centroids
        C[rng.choice(k, g, replace=False)] = C[g]
    lab_o, md_o = helpers.orc_assign(X, C)
    lab, md, _ = km.assign(torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), "fp32", want_mindist=True)
    np.testing.assert_array_equal(lab.cpu().numpy().astype(np.uint32), lab_o)
    # fast-path distances: FP32 products of d terms and the cancellation against ||x||^2 + ||c||^2
    scale = (X.astype(np.float64) ** 2).sum(1) + (C.astype(np.float64) ** 2).sum(1).max()
    assert np.all(np.abs(md.cpu().numpy() - md_o) <= 4 * (d + 4) * 2.0 ** -24 * scale)


@pytest.mark.parametrize("k", [129, 200, 256, 300])
def test_f32_lists_start_again_past_equal_centroids(km, gpu, k):
    """Equal centroids (the zeros of emptied clusters) before a row's own one: they are the
    nearest so far and fill the row's list, and are left behind without a re-score."""
    import torch
    rng = np.random.default_rng(k)
    d, n = 40, 3000
    C = (rng.standard_normal((k, d)) * 20).astype(np.float32)
    C[:30] = 0.0
    own = rng.integers(k // 2, k, n)
    X = (C[own] + 0.1 * rng.standard_normal((n, d))).astype(np.float32)
    lab_o, _ = helpers.orc_assign(X, C)
    np.testing.assert_array_equal(lab_o, own)
    lab, _, refined = km.assign(torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), "fp32", want_mindist=True)
    np.testing.assert_array_equal(lab.cpu().numpy().astype(np.uint32), lab_o)
    assert refined == 0


@pytest.mark.parametrize("k", [64, 130, 256, 300])
def test_f32_two_nearest_within_rounding(km, gpu, k):
    """Rows whose two nearest centroids differ by less than the fast product's rounding, in
    one tile and across tiles: the reference's label, not the fast value's."""
    import torch
    rng = np.random.default_rng(7 * k)
    d, n = 128, 6000
    C = rng.uniform(-10, 10, (k, d)).astype(np.float32)
    a = rng.integers(0, k, n)
    b = (a + rng.integers(1, k, n)) % k
    mid = (C[a].astype(np.float64) + C[b]) / 2
    w = (C[a] - C[b]).astype(np.float64)
    off = rng.uniform(-1, 1, (n, 1)) * 10.0 ** rng.uniform(-9, -6, (n, 1))
    X = (mid + off * w).astype(np.float32)
    lab_o, _ = helpers.orc_assign(X, C)
    lab, _, _ = km.assign(torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), "fp32", want_mindist=True)
    np.testing.assert_array_equal(lab.cpu().numpy().astype(np.uint32), lab_o)
