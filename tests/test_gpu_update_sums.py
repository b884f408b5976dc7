"""The centroid sums at the edges of their batches (128 rows in groups of 32)
and column blocks (32), for rows that allow 16-, 8- and 4-byte copies, against
the oracle's update: the same ordered float sums, so equal bit for bit."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

SIZES = (0, 1, 31, 32, 33, 127, 128, 129, 0, 255, 256, 257, 900, 2500)


@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("d", [1, 2, 3, 4, 30, 31, 32, 33, 34, 36, 64, 97, 130])
def test_update_sums_edges(km, gpu, d, offset):
    import torch
    rng = np.random.default_rng(100 * d + offset)
    lab = rng.permutation(np.repeat(np.arange(len(SIZES)), SIZES)).astype(np.int32)
    n, k = lab.size, len(SIZES)
    X = (rng.standard_normal((n, d)) * rng.choice([1e-3, 1.0, 1e3], (n, 1))).astype(np.float32)
    # `offset` floats into an allocation: rows that start 16-, 8- or 4-byte aligned
    buf = torch.empty(n * d + offset, device=gpu)
    Xd = buf[offset:].view(n, d)
    Xd.copy_(torch.from_numpy(X))
    cen, cnt, perm, off = km.update(Xd, torch.from_numpy(lab).to(gpu), k)
    cen_o, cnt_o = helpers.orc_update(X, lab.astype(np.uint32), k)
    np.testing.assert_array_equal(cen.cpu().numpy().view(np.uint32), cen_o.view(np.uint32))
    np.testing.assert_array_equal(cnt.cpu().numpy().astype(np.uint32), cnt_o)
    np.testing.assert_array_equal(perm.cpu().numpy(), np.argsort(lab, kind="stable"))
    np.testing.assert_array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(SIZES)]))
