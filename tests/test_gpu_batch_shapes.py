"""Batched Lloyd at the edges of its tile shapes (16, 24, 32, 48, 64, 96, 128
centroids; chunks above), row tiles, coordinate stages and of the row count at
which a cluster's sum changes kernel (256), for rows that allow 16-, 8- and
4-byte copies: every instance bit for bit equal to the oracle's single run."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

KS = (1, 2, 16, 17, 24, 25, 32, 33, 48, 49, 64, 65, 96, 97, 128, 129, 192, 193, 256)


@pytest.mark.parametrize("d", [1, 2, 3, 7, 8, 15, 16, 17, 32, 33, 34, 66, 100])
def test_batch_shape_edges(km, gpu, d):
    rng = np.random.default_rng(d)
    shapes, Xs = [], []
    for i, k in enumerate(KS):
        if d * ((k + 31) // 32 * 32) * 4 > 160 * 1024:
            continue
        n = int(rng.choice([63, 64, 65, 127, 129, 255, 257, 511, 513, 2049])) + k * int(rng.choice([1, 3, 40]))
        X, _ = helpers.synth_blobs_np(n, d, max(2, k // 2), -5, 5, 1.0, 1000 * d + i)
        shapes.append((n, d, k))
        Xs.append(X)
    R, seed, tol, maxiter = 2, 11, 1e-4, 12
    b = km.Batch(shapes, restarts=R, seed=seed, tol=tol, maxiter=maxiter).set_data(Xs)
    best, results, _ = b.fit()
    for p, ((n, _, k), X) in enumerate(zip(shapes, Xs)):
        for r in range(R):
            it_o, lab_o, cen_o, ex_o = helpers.orc_lloyd(X, k, tol, seed + p * R + r, maxiter)
            lab, cen = b.instance(p, r)
            np.testing.assert_array_equal(lab, lab_o, err_msg=f"{shapes[p]} restart {r}")
            np.testing.assert_array_equal(cen.view(np.uint32), cen_o.view(np.uint32))
            assert results[p][r][:2] == (it_o, ex_o)
    b.close()


@pytest.mark.parametrize("d", [1, 5, 16, 40])
def test_batch_objective_is_the_cpu_formulas(km, gpu, d):
    """One iteration: the objective is the FP64 sum of the reference's float
    distances to the seeded picks (any order of n < 3000 positive terms: 1e-12)."""
    shapes, Xs = [], []
    for i, k in enumerate((1, 5, 20, 30, 40, 60, 90, 120, 150)):
        X, _ = helpers.synth_blobs_np(1111 + 100 * i, d, k, -5, 5, 1.0, 50 * d + i)
        shapes.append((X.shape[0], d, k))
        Xs.append(X)
    b = km.Batch(shapes, restarts=1, seed=4, maxiter=1).set_data(Xs)
    _, results, _ = b.fit()
    for p, (n, _, k) in enumerate(shapes):
        _, picks = helpers.orc_sample_picks(Xs[p], k, 4 + p)
        _, md = helpers.orc_assign(Xs[p], Xs[p][picks])
        want = float(md.astype(np.float64).sum())
        assert abs(results[p][0][2] - want) <= 1e-12 * want, shapes[p]
    b.close()
