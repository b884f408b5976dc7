"""k > 256: candidate lists whose entries partly fall behind the row's minimum.  A group has g
nearly equal nearest centroids at high indexes and stale ones, each nearer than the last, in
the chunks before, so that a row's list holds kept and dropped entries in every position of
the filter's steps of eight (and is compacted before it overflows): labels equal to the
oracle's for every row."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["bf16", "bf16x3"])
@pytest.mark.parametrize("d", [16, 33, 256])
@pytest.mark.parametrize("stale", [0, 1, 5, 30, 250])
def test_lists_with_stale_entries(km, gpu, prec, d, stale):
    import torch
    rng = np.random.default_rng(100 * d + stale)
    sizes = [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 250, 256, 257]
    base = (rng.standard_normal((len(sizes), d)) * 8).astype(np.float32)
    rows = []
    for s in range(stale):                                # descending distance, the groups side by side
        step = rng.standard_normal((len(sizes), d)) / np.sqrt(d)
        rows.append(base + (3.0 * (stale - s) / stale + 1.0) * step)
    near = [base[g] + 1e-5 * rng.standard_normal((c, d)) for g, c in enumerate(sizes)]
    C = np.concatenate(rows + near).astype(np.float32)
    n = 4500                                              # more rows than centroids
    g = rng.integers(0, len(sizes), n)
    X = (base[g] + 1e-2 * rng.standard_normal((n, d))).astype(np.float32)
    lab_o, _ = helpers.orc_assign(X, C)
    lab, _, refined = km.assign(torch.from_numpy(X).to(gpu), torch.from_numpy(C).to(gpu), prec)
    np.testing.assert_array_equal(lab.cpu().numpy().astype(np.uint32), lab_o)
    assert refined > 0
