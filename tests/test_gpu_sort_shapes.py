"""Label sort at the edges of the one-block form (4096 rows, 256 clusters), of its segments (128 to 1024 rows, 1024 segments) and of the
scan's thread counts: permutation, counts and offsets equal the stable sort's, labels that
leave clusters empty or fill one included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (127, 5), (128, 5), (129, 128), (1000, 129), (4096, 256), (4097, 257),
                                 (5000, 1024), (5000, 1025), (31, 31), (32, 4), (1023, 17), (1024, 33), (1025, 64),
                                 (4095, 100), (4097, 256), (20000, 3), (131072, 40), (131073, 40), (140000, 129),
                                 (262144, 255), (262145, 7), (300001, 513), (524289, 64), (1049000, 11)])
@pytest.mark.parametrize("kind", ["uniform", "skewed", "sorted"])
def test_sort_equals_stable_argsort(km, gpu, n, k, kind):
    import torch
    rng = np.random.default_rng(n + k)
    if kind == "uniform":
        lab = rng.integers(0, k, n)
    elif kind == "skewed":
        lab = np.where(rng.random(n) < 0.9, k - 1, rng.integers(0, max(1, k // 2), n))
    else:
        lab = np.sort(rng.integers(0, k, n))
    X = torch.ones((n, 1), device=gpu)
    _, cnt, perm, off = km.update(X, torch.from_numpy(lab.astype(np.int32)).to(gpu), k)
    ref = np.bincount(lab, minlength=k)
    np.testing.assert_array_equal(cnt.cpu().numpy(), ref)
    np.testing.assert_array_equal(off.cpu().numpy(), np.concatenate([[0], np.cumsum(ref)]))
    np.testing.assert_array_equal(perm.cpu().numpy(), np.argsort(lab, kind="stable"))
