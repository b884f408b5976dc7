"""FP32 kernel matrix at the edges of its 64 x 128 tiles: symmetric builds (the
mirrored half equals the computed one bit for bit), sizes that do and do not allow
16-byte stores, and panels whose rows equal the resident matrix's (through fits)."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("out_bf16", [False, True])
@pytest.mark.parametrize("n,d", [(1, 1), (3, 5), (64, 16), (65, 17), (127, 4), (128, 33), (129, 2), (256, 64), (333, 50),
                                 (516, 12)])
def test_kmat_f32_edges(km, gpu, n, d, out_bf16):
    import torch
    X = torch.from_numpy(helpers.synth_blobs_np(n, d, 3, -1, 1, 0.5, n + d)[0]).to(gpu)
    for kind, p in (("linear", {}), ("polynomial", dict(gamma=0.5, coef=1.0, degree=3)), ("gaussian", dict(sigma=2.0))):
        K, dg = km.kernel_matrix(X, kernel=kind, precision="fp32", out_bf16=out_bf16, want_diag=True, **p)
        Xd = X.double()
        G = Xd @ Xd.T
        sq = (Xd * Xd).sum(1)
        ref = G if kind == "linear" else (0.5 * G + 1.0) ** 3 if kind == "polynomial" else \
            (-(sq[:, None] + sq[None] - 2 * G).clamp_min(0) / 8.0).exp()
        # FP32 products of d terms, three more operations (degree 3: relative 3x), BF16 storage
        arg = 0.5 * G.abs().max() + 1.0 + sq.max()
        lim = (d + 16) * 2.0 ** -23 * float(arg) * 3 * max(1.0, float(ref.abs().max() / arg)) + \
            (2.0 ** -8 * float(ref.abs().max()) if out_bf16 else 0.0)
        assert float((K.double() - ref).abs().max()) <= lim
        assert torch.equal(K, K.T)
        assert torch.equal(torch.diagonal(K).float(), dg.to(K.dtype).float())


@pytest.mark.parametrize("panel", [1, 63, 64, 100, 200])
def test_kmat_f32_panels_equal_resident(km, gpu, panel):
    X, _ = helpers.synth_blobs_np(333, 7, 4, -1, 1, 0.6, 9)
    out = []
    for pr in (0, panel):
        m = km.KernelKMeans(333, 7, 5, kernel="polynomial", gamma=0.2, precision="fp32", maxiter=6, panel_rows=pr).set_data(X)
        out.append(m.fit())
        m.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert out[0][1].score == out[1][1].score
