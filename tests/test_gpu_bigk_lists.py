"""k > 256: rows whose candidates overflow the chunked kernel's lists (more than
256) go through the FP32 pass with its own lists.  Groups of 300 centroids at
spreads from far above to far below the near-tie windows (single BF16, split and
FP32) leave such rows with one, a few, up to 256 and more candidates: labels equal
to the oracle's for every row."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
@pytest.mark.parametrize("d,k,n", [(64, 700, 3000), (20, 1300, 1501), (33, 400, 777), (130, 2100, 2200)])
def test_overflowing_candidate_lists(km, gpu, prec, d, k, n):
    import torch
    rng = np.random.default_rng(7 * d + k)
    groups = max(1, k // 300)
    base = (rng.standard_normal((groups, d)) * 4).astype(np.float32)
    spread = np.array([1e-1, 3e-3, 1e-3, 1e-4, 1e-6, 1.0, 0.0], np.float32)
    owner = rng.integers(0, groups, k)
    C = (base[owner] + spread[owner % 7][:, None] * rng.standard_normal((k, d))).astype(np.float32)
    g = rng.integers(0, groups, n)
    X = (base[g] + rng.choice([1e-3, 1e-1, 1.0], (n, 1)) * rng.standard_normal((n, d))).astype(np.float32)
    lab_o, _ = helpers.orc_assign(X, C)
    lab, _, refined = km.assign(torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), prec, want_mindist=True)
    np.testing.assert_array_equal(lab.cpu().numpy().astype(np.uint32), lab_o)
    assert refined > 0


@pytest.mark.parametrize("d", [15, 16, 63, 64, 65, 79, 80, 127, 128, 129, 192, 256])
def test_runs_of_the_fp32_pass(km, gpu, d):
    """The FP32 pass sums its products in runs of 64 coordinates and narrows its near-tie
    window accordingly: centroids closer to one another than the window for the whole
    chain, at the edges of the runs."""
    import torch
    rng = np.random.default_rng(d)
    k, n = 600, 1000
    base = (rng.standard_normal(d) * 6).astype(np.float32)
    C = (base + 1e-3 * rng.standard_normal((k, d))).astype(np.float32)
    X = (base + rng.choice([1e-4, 1e-3, 1e-2], (n, 1)) * rng.standard_normal((n, d))).astype(np.float32)
    lab_o, md_o = helpers.orc_assign(X, C)
    lab, _, refined = km.assign(torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), "bf16x3", want_mindist=True)
    np.testing.assert_array_equal(lab.cpu().numpy().astype(np.uint32), lab_o)
    assert refined > 0


@pytest.mark.parametrize("d", [4, 5, 12, 64, 124, 128, 132, 200, 256])
@pytest.mark.parametrize("sizes", [(5,) * 60, (5, 6, 7, 8, 31, 32, 33, 63, 64, 65, 100, 255, 256), (16, 256, 5, 250, 9)])
def test_wide_rows(km, gpu, d, sizes):
    """Rows with 5..256 candidates, of groups of equal and of nearly equal centroids, many
    and few in a segment, over the passes of 32 pairs and of 8 rows."""
    import torch
    rng = np.random.default_rng(d + len(sizes))
    base = (rng.standard_normal((len(sizes), d)) * 5).astype(np.float32)
    C = np.repeat(base, sizes, axis=0)
    C = np.where(rng.random((len(C), 1)) < 0.5, C, C + 1e-5 * rng.standard_normal(C.shape)).astype(np.float32)
    C = C[rng.permutation(len(C))]
    n = 1500
    g = rng.integers(0, len(sizes), n)
    X = (base[g] + 1e-2 * rng.standard_normal((n, d))).astype(np.float32)
    X[::3] = rng.standard_normal((len(X[::3]), d)) * 5                # rows of other queues between
    lab_o, md_o = helpers.orc_assign(X, C)
    lab, md, refined = km.assign(torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), "bf16x3", want_mindist=True)
    np.testing.assert_array_equal(lab.cpu().numpy().astype(np.uint32), lab_o)
    assert refined > 0
