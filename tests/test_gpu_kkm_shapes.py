"""One kernel k-means iteration and the tensor-core kernel matrix at the edges of their
tiles.  The points are small whole numbers, so the linear kernel's values, and their sums
per cluster, are exact in FP32 (and in BF16: at most 64 in size) whatever the order: what
is left to differ from FP64 is the rounding of -2 E/|c| + ctilde."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, d, seed):
    return np.random.default_rng(seed).integers(-4, 5, (n, d)).astype(np.float32)


# V.K takes four columns a lane (n % 4 == 0) in pairs of batches of 1024 (FP32) or 1536
# (BF16) columns, else one column a lane; clusters are reduced 32 at a time; ctilde takes
# 1024 of a cluster's rows a step.
@pytest.mark.parametrize("k_bf16", [False, True])
@pytest.mark.parametrize("n,k,skew", [(5, 1, 0), (127, 31, 0), (128, 32, 0), (1020, 33, 0), (1024, 5, 0), (1028, 5, 0),
                                      (1536, 64, 0), (2048, 7, 1), (2052, 256, 0), (3072, 3, 1), (3076, 3, 1), (3077, 40, 0)])
def test_kkm_iteration_vs_fp64(km, gpu, n, k, skew, k_bf16):
    X = _points(n, 4, n + k)
    lab0 = np.random.default_rng(n).integers(0, k, n).astype(np.uint32)
    if skew:
        lab0[: n - 3] = k // 2                       # one large cluster, some empty or tiny
    m = km.KernelKMeans(n, 4, k, kernel="linear", maxiter=1, precision="fp32", k_bf16=k_bf16).set_data(X)
    lab, r = m.fit(init_labels=lab0)
    m.close()
    Xd = X.astype(np.float64)
    V = np.zeros((k, n))
    V[lab0, np.arange(n)] = 1.0
    E = Xd @ (V @ Xd).T                              # (n, k)
    cnt = V.sum(1)
    ct = np.array([E[lab0 == c, c].sum() / max(cnt[c], 1) ** 2 for c in range(k)])
    inv = np.divide(-2.0, cnt, out=np.zeros(k), where=cnt > 0)
    D = inv * E + np.where(ct == 0, np.inf, ct)
    tol = 4 * 2.0 ** -24 * (np.abs(inv * E) + np.where(ct == 0, 0.0, np.abs(ct))).max()
    best = D.min(1)
    assert (D[np.arange(n), lab] <= best + 2 * tol).all()
    assert abs(r.score - best.sum()) <= n * tol


@pytest.mark.parametrize("precision", ["bf16", "bf16x3"])
@pytest.mark.parametrize("out_bf16", [False, True])
@pytest.mark.parametrize("n,d", [(1, 4), (63, 16), (127, 64), (128, 65), (129, 3), (255, 64), (256, 130), (257, 8), (388, 64),
                                 (515, 40)])
def test_kmat_tensor_core_edges(km, gpu, n, d, out_bf16, precision):
    """Whole numbers below 2^24 come out of the tensor cores and both epilogues exactly
    (stored as BF16: rounded once)."""
    import torch
    X = torch.from_numpy(_points(n, d, n * d)).to(gpu)
    G = X.double() @ X.double().T
    for kind, p, ref in (("linear", {}, G), ("polynomial", dict(gamma=1.0, coef=1.0, degree=2), (G + 1) ** 2)):
        K, dg = km.kernel_matrix(X, kernel=kind, precision=precision, out_bf16=out_bf16, want_diag=True, **p)
        assert torch.equal(K, ref.float().to(K.dtype))
        assert torch.equal(dg, torch.diagonal(ref).float())
