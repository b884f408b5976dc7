"""Centroid sums where most clusters are small (a warp each) and a few are large (the ring):
sizes at the edges of both (0, 1, 31..33, 255..257 rows, thousands), clusters up to and
beyond the 1024 that are sorted by size, every row alignment.  Centroids bit for bit the
oracle's; the objective against FP64 (runs of 16 FP32 terms, each term with one more
rounding: 18 * 2^-24 of a sum of positive terms)."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 1000, 5000]


def _labels(k, rng):
    counts = np.full(k, 40)
    counts[rng.permutation(k)[: len(SIZES)]] = SIZES
    lab = np.repeat(np.arange(k, dtype=np.uint32), counts)
    return lab[rng.permutation(len(lab))]


@pytest.mark.parametrize("d", [1, 2, 3, 4, 32, 33, 64, 100])
@pytest.mark.parametrize("k", [700, 1024, 1025, 3000])
def test_update_with_small_and_large_clusters(km, gpu, k, d):
    import torch
    rng = np.random.default_rng(k + d)
    lab = _labels(k, rng)
    X = rng.standard_normal((len(lab), d)).astype(np.float32)
    cen_o, cnt_o = helpers.orc_update(X, lab, k)
    C, cnt, _, off = km.update(torch.from_numpy(X).to(gpu), torch.from_numpy(lab.astype(np.int32)).to(gpu), k)
    np.testing.assert_array_equal(C.cpu().numpy().view(np.uint32), cen_o.view(np.uint32))
    np.testing.assert_array_equal(cnt.cpu().numpy().astype(np.uint32), np.bincount(lab, minlength=k))
    np.testing.assert_array_equal(off.cpu().numpy()[1:], np.cumsum(np.bincount(lab, minlength=k)))


@pytest.mark.parametrize("d", [3, 32, 50])
@pytest.mark.parametrize("k", [1024, 1500])
def test_fit_with_small_clusters(km, gpu, k, d):
    rng = np.random.default_rng(k * d)
    base = rng.standard_normal((k, d)).astype(np.float32) * 20
    lab = _labels(k, rng)
    X = (base[lab] + 0.1 * rng.standard_normal((len(lab), d))).astype(np.float32)
    m = km.Lloyd(len(X), d, k, init="given", maxiter=2, conv="none", precision="fp32").set_data(X)
    got, cen, r = m.fit(base)
    m.close()
    _, lab_o, cen_o, _ = helpers.orc_lloyd(X, k, 0.0, 0, 2, C0=base)
    np.testing.assert_array_equal(got, lab_o)
    np.testing.assert_array_equal(cen.view(np.uint32), cen_o.view(np.uint32))
    _, _, before, _ = helpers.orc_lloyd(X, k, 0.0, 0, 1, C0=base)
    want = ((X.astype(np.float64) - before.astype(np.float64)[got]) ** 2).sum()
    assert abs(r.objective - want) <= 18 * 2.0 ** -24 * want


@pytest.mark.parametrize("d", [3, 32, 50])
@pytest.mark.parametrize("k", [700, 1024])
def test_noalloc_update_with_small_and_large_clusters(km, gpu, k, d):
    import torch
    rng = np.random.default_rng(k - d)
    lab = _labels(k, rng)
    X = rng.standard_normal((len(lab), d)).astype(np.float32)
    Xd, ld = torch.from_numpy(X).to(gpu), torch.from_numpy(lab.astype(np.int32)).to(gpu)
    C, cnt = torch.empty((k, d), device=gpu), torch.empty(k, dtype=torch.int32, device=gpu)
    km.check(km.lib().km_update_noalloc(Xd.data_ptr(), ld.data_ptr(), len(lab), d, k, C.data_ptr(), cnt.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream), "km_update_noalloc")
    cen_o, _ = helpers.orc_update(X, lab, k)
    np.testing.assert_array_equal(C.cpu().numpy().view(np.uint32), cen_o.view(np.uint32))
    np.testing.assert_array_equal(cnt.cpu().numpy().astype(np.uint32), np.bincount(lab, minlength=k))


@pytest.mark.parametrize("d", [1, 3, 6, 33, 50])
@pytest.mark.parametrize("k,rows", [(5, 31), (60, 20), (127, 31), (127, 33), (256, 63), (256, 65), (500, 60)])
def test_update_of_few_small_clusters(km, gpu, k, rows, d):
    import torch
    rng = np.random.default_rng(k * rows + d)
    n = k * rows
    lab = rng.integers(0, k, n).astype(np.uint32)
    X = rng.standard_normal((n, d)).astype(np.float32)
    cen_o, _ = helpers.orc_update(X, lab, k)
    C, cnt, _, _ = km.update(torch.from_numpy(X).to(gpu), torch.from_numpy(lab.astype(np.int32)).to(gpu), k)
    np.testing.assert_array_equal(C.cpu().numpy().view(np.uint32), cen_o.view(np.uint32))
    np.testing.assert_array_equal(cnt.cpu().numpy().astype(np.uint32), np.bincount(lab, minlength=k))
