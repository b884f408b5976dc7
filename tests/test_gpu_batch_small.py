"""Batches of small problems run a CTA an instance; one instance too many rows for that
sends the whole batch through the tiles.  Either way every instance is bit for bit the
oracle's single run, and the objective is the same in both (its order is fixed).  Sizes at
the edges of the kernel: chunks of 8, 16 and 32 centroids, warps with one and two groups
of 32 rows, sums by a warp (k * d <= 24, d <= 8) and by a thread, 16-byte rows and others."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (2, 1, 2), (31, 2, 3), (32, 3, 8), (33, 8, 3), (100, 12, 2), (100, 5, 5), (255, 4, 8), (256, 9, 9),
          (257, 16, 16), (300, 1, 17), (511, 7, 32), (513, 20, 33), (700, 6, 64), (1000, 2, 65), (1025, 64, 4),
          (300, 1, 256), (2000, 8, 32), (4100, 3, 8)]


@pytest.mark.parametrize("tol,maxiter", [(1e-4, 15), (0.0, 1), (1e30, 300)])
def test_small_batch_equals_oracle_and_tiles(km, gpu, tol, maxiter):
    Xs = [helpers.synth_blobs_np(n, d, max(2, k // 2), -5, 5, 1.0, 10 * i)[0] for i, (n, d, k) in enumerate(SHAPES)]
    Xs[5][:] = Xs[5][0]                      # all rows equal but one: emptied clusters
    Xs[5][7] += 1.0
    R, seed = 2, 5
    big = (20000, 40, 4)
    Xb, _ = helpers.synth_blobs_np(*big, -5, 5, 1.0, 999)
    got = []
    for shapes, data in ((SHAPES, Xs), (SHAPES + [big], Xs + [Xb])):
        b = km.Batch(shapes, restarts=R, seed=seed, tol=tol, maxiter=maxiter).set_data(data)
        for _ in range(2):                   # a second fit starts from the same picks
            _, results, _ = b.fit()
        got.append((results[: len(SHAPES)], [b.instance(p, r) for p in range(len(SHAPES)) for r in range(R)]))
        b.close()
    (small, inst), (tiles, inst_t) = got
    assert small == tiles
    for p, ((n, _, k), X) in enumerate(zip(SHAPES, Xs)):
        for r in range(R):
            it_o, lab_o, cen_o, ex_o = helpers.orc_lloyd(X, k, tol, seed + p * R + r, maxiter)
            assert small[p][r][:2] == (it_o, ex_o), (SHAPES[p], r)
            for lab, cen in (inst[p * R + r], inst_t[p * R + r]):
                np.testing.assert_array_equal(lab, lab_o, err_msg=f"{SHAPES[p]} restart {r}")
                np.testing.assert_array_equal(cen.view(np.uint32), cen_o.view(np.uint32))


def test_many_instances_of_few_columns(km, gpu):
    """More instances than SMs, rows enough for the tiles but d <= 3: a CTA each."""
    shapes = [(9000 + i, 1 + i % 3, 40) for i in range(160)]
    Xs = [helpers.synth_blobs_np(n, d, 20, -50, 50, 1.0, i)[0] for i, (n, d, _) in enumerate(shapes)]
    b = km.Batch(shapes, restarts=1, seed=3, maxiter=4).set_data(Xs)
    b.fit()
    for p in range(0, 160, 13):
        _, lab_o, cen_o, _ = helpers.orc_lloyd(Xs[p], 40, 1e-4, 3 + p, 4)
        lab, cen = b.instance(p, 0)
        np.testing.assert_array_equal(lab, lab_o)
        np.testing.assert_array_equal(cen.view(np.uint32), cen_o.view(np.uint32))
    b.close()
