"""V.K of a BF16 kernel matrix at the edges of its batches: 1792 columns (14 loads of four
columns a lane), summed in pairs of 3584, so that a row has one, two and three batches and
more than a pair.  Whole-numbered points keep every value and sum exact in BF16 and FP32;
what is left to differ from FP64 is the rounding of -2 E/|c| + ctilde."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 7, 40])
@pytest.mark.parametrize("n", [1788, 1792, 1796, 3580, 3584, 3588, 5376, 5380, 7168, 7172])
def test_bf16_batches_vs_fp64(km, gpu, n, k):
    rng = np.random.default_rng(n + k)
    X = rng.integers(-4, 5, (n, 4)).astype(np.float32)
    lab0 = rng.integers(0, k, n).astype(np.uint32)
    m = km.KernelKMeans(n, 4, k, kernel="linear", maxiter=1, precision="fp32", k_bf16=True).set_data(X)
    lab, r = m.fit(init_labels=lab0)
    m.close()
    Xd = X.astype(np.float64)
    S = np.stack([Xd[lab0 == c].sum(0) for c in range(k)])     # E = X S^T
    E = Xd @ S.T
    cnt = np.bincount(lab0, minlength=k).astype(np.float64)
    ct = np.array([E[lab0 == c, c].sum() / max(cnt[c], 1) ** 2 for c in range(k)])
    inv = np.divide(-2.0, cnt, out=np.zeros(k), where=cnt > 0)
    ok = np.where(ct == 0, 0.0, ct)
    D = inv * E + np.where(ct == 0, np.inf, ct)
    tol = 4 * 2.0 ** -24 * (np.abs(inv * E) + np.abs(ok)).max()
    best = D.min(1)
    assert (D[np.arange(n), lab] <= best + 2 * tol).all()
    assert abs(r.score - best.sum()) <= n * tol
