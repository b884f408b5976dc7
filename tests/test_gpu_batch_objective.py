"""The objective of a batched instance does not depend on the tile variant in use: it is
the FP64 sum, in a fixed order, of the reference's float distances.  The order is that of
km.h: blocks of 32 rows, each by the tree r + (r ^ 16), ^ 8, .. ^ 1; of the blocks, lane l
adds l, l + 32, ... and the lanes are added by the same tree."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


def _tree(v):
    """32 values along the last axis, added as lanes that exchange by xor."""
    v = v.copy()
    for o in (16, 8, 4, 2, 1):
        v = v + v[..., np.arange(32) ^ o]
    return v[..., 0]


def _ordered_sum(md):
    v = np.zeros((len(md) + 31) // 32 * 32)
    v[: len(md)] = md.astype(np.float64)
    blocks = _tree(v.reshape(-1, 32))
    lanes = np.zeros(32)
    for b in range(0, len(blocks), 32):
        part = blocks[b:b + 32]
        lanes[: len(part)] += part
    return float(_tree(lanes))


def test_objective_in_a_fixed_order_for_every_variant(km, gpu):
    shapes, Xs = [], []
    for i, (d, k) in enumerate([(3, 1), (8, 16), (16, 20), (5, 32), (33, 40), (20, 64), (64, 70), (10, 128), (7, 200)]):
        X, _ = helpers.synth_blobs_np(1500 + 731 * i, d, max(k, 2), -5, 5, 1.0, 70 + i)
        # rows of very different lengths: the sums round, so their order shows
        X *= 10.0 ** np.random.default_rng(i).uniform(-4, 4, (X.shape[0], 1)).astype(np.float32)
        shapes.append((X.shape[0], d, k))
        Xs.append(X)
    R, seed = 2, 9
    b = km.Batch(shapes, restarts=R, seed=seed, maxiter=1).set_data(Xs)
    want = []
    for p, (_, _, k) in enumerate(shapes):
        for r in range(R):
            _, picks = helpers.orc_sample_picks(Xs[p], k, seed + p * R + r)
            _, md = helpers.orc_assign(Xs[p], Xs[p][picks])
            want.append(_ordered_sum(md))
    for tuned in (False, True):
        if tuned:
            b.tune()
        best, results, _ = b.fit()
        assert [results[p][r][2] for p in range(len(shapes)) for r in range(R)] == want, f"tuned {tuned}"
        for p in range(len(shapes)):
            r = int(np.argmin(want[p * R:(p + 1) * R]))
            np.testing.assert_array_equal(best[p][0], b.instance(p, r)[0])
    b.close()
