"""Timed cases of the framework's public Python entry points (km.py).

listed() holds one case per kind of work a program asks for: fits of Lloyd
k-means (small, ordinary, ragged, the n = 1M benchmark and the very-large-k
benchmark), seeding, assignment of points to given centroids, the centroid
update alone, kernel k-means, the kernel matrix alone and batched problems.
draw() gives further cases over the same ranges.  Inputs are seeded Gaussian
blobs, as in the benchmark and the tests, made on the GPU.
"""
from __future__ import annotations

import importlib.util
import math
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]


def _load_km():
    spec = importlib.util.spec_from_file_location("km_gb300", ROOT / "matrix-centric-k-means_gb300" / "km.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


km = _load_km()


def listed():
    return [
        # The smallest fit: a digits-sized table of integer features in host
        # memory, run the way the Kmeans class runs its linear kernel (labels
        # i % k first, emptied clusters excluded, stop on the score).  Latency
        # and launches are all there is.
        dict(name="fit_digits", kind="fit", n=1797, d=64, k=10, precision="bf16x3", init="round_robin",
             empty="exclude", conv="score", tol=1e-4, maxiter=100, data="digits", where="host"),
        # The headline workload of the benchmark: 20 iterations at n = 1M.
        dict(name="fit_1m", kind="fit", n=1048576, d=128, k=256, precision="bf16x3", init="given", empty="zero",
             conv="none", tol=1e-4, maxiter=20, data="separated", where="device"),
        # An ordinary table in the handle's default precision and stop rule.
        dict(name="fit_fp32", kind="fit", n=200000, d=100, k=64, precision="fp32", init="given", empty="zero",
             conv="shift", tol=1e-4, maxiter=20, data="overlapping", where="device"),
        # Ragged sizes in every dimension (d not a multiple of 4, so rows are
        # not 16-byte aligned), single-BF16 operands.
        dict(name="fit_ragged", kind="fit", n=300007, d=50, k=37, precision="bf16", init="given", empty="zero",
             conv="none", tol=1e-4, maxiter=10, data="overlapping", where="device"),
        # The largest: 4M BF16-stored points in Zipf-sized clusters, k = 4096
        # (the benchmark's very-large-k workload), seeded sample picks.
        dict(name="fit_bigk", kind="fit", n=4194304, d=256, k=4096, precision="bf16x3", init="sample", empty="zero",
             conv="none", tol=1e-5, maxiter=2, data="zipf_bf16", where="device"),
        # Seeding alone: greedy k-means++.
        dict(name="seed_plusplus", kind="seed", n=262144, d=32, k=100, data="overlapping"),
        # New points against trained centroids: the prediction step of a server.
        dict(name="assign", kind="assign", n=65536, d=64, k=128, precision="bf16x3", data="overlapping"),
        # The centroid update alone, ragged row length.
        dict(name="update", kind="update", n=500000, d=30, k=100, data="overlapping"),
        # Kernel k-means as the Kmeans class runs it: FP32 kernel matrix, K
        # resident, stop on the score.
        dict(name="kernel_fit_fp32", kind="kernel_fit", n=20000, d=64, k=20, kernel="polynomial", precision="fp32",
             k_bf16=False, panel="auto", check=True, maxiter=20),
        # Kernel k-means at the benchmark's size: tensor-core kernel matrix of
        # 16 GiB, then iterations that stream it.
        dict(name="kernel_fit_64k", kind="kernel_fit", n=65536, d=512, k=64, kernel="polynomial",
             precision="bf16x3", k_bf16=False, panel="resident", check=False, maxiter=10),
        # The kernel matrix alone (for a program with its own solver).
        dict(name="kernel_matrix", kind="kernel_matrix", n=24000, d=200, kernel="gaussian", precision="bf16x3",
             k_bf16=False),
        # Many small independent problems, several restarts each, one launch.
        dict(name="batch", kind="batch", problems=64, restarts=4, nlo=1024, nhi=65536, maxiter=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "fit", "seed", "assign", "update", "kernel_fit", "kernel_fit",
                       "kernel_matrix", "batch"])
    precision = rng.choice(["fp32", "bf16", "bf16x3"])
    if kind == "fit":
        d = _log(rng, 2, 512)
        large = rng.random() < 0.25 and d <= 320
        k = _log(rng, 257, 2048) if large else _log(rng, 2, 256)
        top = 2.0e11 if large else 6.0e11                     # bounds n * d * k of one iteration
        n = _log(rng, 1500, max(2000, min(2000000, int(top / (d * k)))))
        k = min(k, n // 8)
        return dict(kind=kind, n=n, d=d, k=k, precision=precision,
                    init=rng.choice(["given", "given", "sample", "round_robin"]),
                    empty=rng.choice(["zero", "exclude"]), conv=rng.choice(["none", "shift", "score"]), tol=1e-4,
                    maxiter=rng.randint(2, 12), data=rng.choice(["separated", "overlapping"]),
                    where=rng.choice(["device", "device", "host"]) if n * d < 40000000 else "device")
    if kind == "seed":
        return dict(kind=kind, n=_log(rng, 2000, 400000), d=_log(rng, 2, 256), k=_log(rng, 4, 160),
                    data="overlapping")
    if kind == "assign":
        d = _log(rng, 2, 512)
        return dict(kind=kind, n=_log(rng, 200, 1000000), d=d, k=_log(rng, 2, 190), precision=precision,
                    data="overlapping")
    if kind == "update":
        return dict(kind=kind, n=_log(rng, 1000, 1500000), d=_log(rng, 2, 256), k=_log(rng, 2, 500),
                    data="overlapping")
    if kind == "kernel_fit":
        panel = rng.choice(["auto", "resident", "fused", "panel"])
        if panel == "fused" and precision == "fp32":
            precision = "bf16x3"
        return dict(kind=kind, n=_log(rng, 1500, 40000), d=_log(rng, 4, 512), k=_log(rng, 2, 100),
                    kernel=rng.choice(["polynomial", "gaussian", "linear", "sigmoid"]), precision=precision,
                    k_bf16=precision == "bf16" and rng.random() < 0.5, panel=panel, check=rng.random() < 0.5,
                    maxiter=rng.randint(2, 12))
    if kind == "kernel_matrix":
        return dict(kind=kind, n=_log(rng, 500, 32000), d=_log(rng, 4, 512),
                    kernel=rng.choice(["polynomial", "gaussian", "linear", "sigmoid"]), precision=precision,
                    k_bf16=precision == "bf16" and rng.random() < 0.5)
    return dict(kind=kind, problems=_log(rng, 8, 64), restarts=rng.randint(1, 8), nlo=512, nhi=_log(rng, 4096, 40000),
                maxiter=rng.randint(10, 40))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + 17)
    return g


def _blobs(n, d, blobs, lo, hi, sigma, g, zipf=0.0):
    """(points, blob of each point) on the GPU; sigma a number or a per-blob tensor."""
    centers = torch.rand((blobs, d), generator=g, device="cuda") * (hi - lo) + lo
    if zipf > 0:
        w = torch.arange(1, blobs + 1, device="cuda", dtype=torch.float64).pow(-zipf).cumsum(0)
        u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * w[-1]
        lab = torch.searchsorted(w, u).clamp_(max=blobs - 1)
    else:
        lab = torch.randint(blobs, (n,), generator=g, device="cuda")
    X = torch.empty((n, d), device="cuda")
    step = max(1, (1 << 28) // d)
    for a in range(0, n, step):
        part = X[a:a + step]
        part.normal_(generator=g)
        part.mul_(sigma[lab[a:a + step], None] if isinstance(sigma, torch.Tensor) else sigma)
        part.add_(centers[lab[a:a + step]])
    return X, lab


def _points(case, g):
    n, d, k = case["n"], case["d"], case["k"]
    data = case["data"]
    if data == "digits":                  # integer features in [0, 16]
        X, lab = _blobs(n, d, k, 0.0, 16.0, 3.0, g)
        return X.round_().clamp_(0, 16), lab
    if data == "separated":
        return _blobs(n, d, k, -10.0, 10.0, 1.0, g)
    if data == "zipf_bf16":
        sigma = torch.rand(k, generator=g, device="cuda") * 1.8 + 0.2
        X, lab = _blobs(n, d, k, -20.0, 20.0, sigma, g, zipf=1.1)
        return X.to(torch.bfloat16), lab
    return _blobs(n, d, k, -3.0, 3.0, 1.5, g)


def _kernel_points(case, g):
    blobs = case.get("k", 32)
    return _blobs(case["n"], case["d"], blobs, -1.0, 1.0, 0.25, g)[0]


def _kernel_args(case):
    d = case["d"]
    return {"polynomial": dict(gamma=1.0 / d, coef=1.0, degree=2), "gaussian": dict(sigma=math.sqrt(d) / 8.0),
            "sigmoid": dict(gamma=1.0 / d, coef=1.0), "linear": {}}[case["kernel"]]


def _picked_rows(X, k, seed):
    rows = np.random.default_rng(seed).choice(X.shape[0], k, replace=False)
    return X[torch.from_numpy(np.sort(rows)).cuda()].float()


def _batch_shapes(case, seed):
    # the shapes belong to the case, the points to the seed
    rng = np.random.default_rng(case["problems"] * 7 + case["restarts"])
    shapes = []
    for _ in range(case["problems"]):
        n = int(np.exp(rng.uniform(np.log(case["nlo"]), np.log(case["nhi"]))))
        d = int(rng.choice([2, 8, 16, 32, 64, 128, 256]))
        shapes.append((n, d, min(int(rng.integers(2, 129)), n - 1)))
    return shapes


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "fit":
        X, _ = _points(case, g)
        s["C0"] = _picked_rows(X, case["k"], seed).cpu().numpy() if case["init"] == "given" else None
        s["X"] = X.cpu().numpy() if case["where"] == "host" else X
        s["m"] = km.Lloyd(case["n"], case["d"], case["k"], tol=case["tol"], seed=1, maxiter=case["maxiter"],
                          init=case["init"], precision=case["precision"], conv=case["conv"], empty=case["empty"])
    elif kind == "seed":
        X, _ = _points(case, g)
        s["m"] = km.Lloyd(case["n"], case["d"], case["k"], seed=1, init="plusplus", precision="fp32").set_data(X)
    elif kind == "assign":
        s["X"], _ = _points(case, g)
        s["C"] = _picked_rows(s["X"], case["k"], seed) * 0.9
    elif kind == "update":
        s["X"], lab = _points(case, g)
        s["labels"] = lab.to(torch.int32)
    elif kind == "kernel_fit":
        s["X"] = _kernel_points(case, g)
        n = case["n"]
        panel = {"auto": "auto", "resident": 0, "fused": "fused", "panel": max(1, n // 3)}[case["panel"]]
        s["m"] = km.KernelKMeans(n, case["d"], case["k"], kernel=case["kernel"], tol=1e-4, maxiter=case["maxiter"],
                                 precision=case["precision"], k_bf16=case["k_bf16"], check_converged=case["check"],
                                 panel_rows=panel, **_kernel_args(case))
    elif kind == "kernel_matrix":
        s["X"] = _kernel_points(case, g)
    else:
        shapes = _batch_shapes(case, seed)
        Xs = [_blobs(n, d, k, -5.0, 5.0, 1.0, g)[0].cpu().numpy() for n, d, k in shapes]
        s["m"] = km.Batch(shapes, restarts=case["restarts"], seed=3, tol=1e-4, maxiter=case["maxiter"]).set_data(Xs)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "fit":
        m = s["m"]
        if case["data"] == "zipf_bf16":
            m.set_data_bf16(s["X"])
        else:
            m.set_data(s["X"])
        labels, centroids, r = m.fit(s["C0"])
        return {"labels": labels.view(np.int32), "centroids": centroids, "iterations": int(r.iterations),
                "converged_iter": int(r.converged_iter), "objective": float(r.objective)}
    if kind == "seed":
        return {"centroids": s["m"].init_centroids()}
    if kind == "assign":
        labels, mindist, _ = km.assign(s["X"], s["C"], precision=case["precision"], want_mindist=True)
        return {"labels": labels, "mindist": mindist}
    if kind == "update":
        centroids, counts, perm, offsets = km.update(s["X"], s["labels"], case["k"])
        return {"centroids": centroids, "counts": counts, "perm": perm, "offsets": offsets}
    if kind == "kernel_fit":
        labels, r = s["m"].set_data(s["X"]).fit()
        return {"labels": labels.view(np.int32), "iterations": int(r.iterations), "score": float(r.score)}
    if kind == "kernel_matrix":
        K, diag = km.kernel_matrix(s["X"], kernel=case["kernel"], precision=case["precision"],
                                   out_bf16=case["k_bf16"], want_diag=True, **_kernel_args(case))
        return {"K": K, "diag": diag}
    best, results, _ = s["m"].fit()
    return {"labels": np.concatenate([b[0] for b in best]).view(np.int32),
            "centroids": np.concatenate([b[1].ravel() for b in best]),
            "iterations": np.array([[r[1] for r in p] for p in results]),
            "objective": np.array([[r[2] for r in p] for p in results])}


# ---------------------------------------------------------------------------
# The least work of a pass
# ---------------------------------------------------------------------------
BATCH_ITERS = 15   # iterations a batched instance is counted with (it stops by itself, most of them near here)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        fl = by = 0
        for n, d, k in _batch_shapes(case, 0):
            it = min(BATCH_ITERS, case["maxiter"])
            fl += case["restarts"] * it * 3.0 * n * d * k
            by += n * d * 4 + n * 4 + k * d * 4
        return {"bytes": by, "flops": fl}
    n, d = case["n"], case["d"]
    if kind == "fit":
        k = case["k"]
        # a fit that stops by itself is counted with a tenth of its budget
        it = case["maxiter"] if case["conv"] == "none" else max(2, case["maxiter"] // 10)
        x = n * d * (2 if case["data"] == "zipf_bf16" else 4)
        return {"bytes": it * (x + 4.0 * n + 8.0 * k * d), "flops": it * 2.0 * n * d * k}
    if kind == "seed":
        k = case["k"]
        cand = 2 + math.ceil(math.log(k))
        return {"bytes": (k - 1) * (4.0 * n * d + 8.0 * n), "flops": (k - 1) * 3.0 * n * d * cand}
    if kind == "assign":
        k = case["k"]
        return {"bytes": 4.0 * n * d + 8.0 * n + 4.0 * k * d, "flops": 2.0 * n * d * k}
    if kind == "update":
        return {"bytes": 4.0 * n * d + 8.0 * n + 4.0 * case["k"] * d, "flops": 1.0 * n * d}
    ksize = 2 if case["k_bf16"] else 4
    if kind == "kernel_matrix":
        return {"bytes": 4.0 * n * d + ksize * float(n) * n, "flops": float(n) * n * d}
    it = case["maxiter"] if not case["check"] else max(2, case["maxiter"] // 4)
    if case["panel"] == "fused":
        return {"bytes": it * 8.0 * n * d, "flops": it * 2.0 * n * n * d}
    return {"bytes": 4.0 * n * d + ksize * float(n) * n * (1 + it), "flops": float(n) * n * d}


# ---------------------------------------------------------------------------
# The same results in 64 bits
# ---------------------------------------------------------------------------

def _assign64(X, C, dead):
    """(labels, smallest squared distance) of FP64 points."""
    n = X.shape[0]
    lab = torch.empty(n, dtype=torch.int64, device="cuda")
    best = torch.empty(n, dtype=torch.float64, device="cuda")
    c2 = (C * C).sum(1)
    if dead is not None:
        c2 = torch.where(dead, torch.full_like(c2, math.inf), c2)
    step = max(1, (1 << 27) // max(C.shape[0], X.shape[1]))
    for a in range(0, n, step):
        x = X[a:a + step]
        v = torch.addmm(c2[None, :].expand(x.shape[0], -1), x, C.T, alpha=-2.0)
        m, i = v.min(1)
        lab[a:a + step] = i
        best[a:a + step] = ((x - C[i]) ** 2).sum(1)
    return lab, best


def _means64(X, lab, k):
    cnt = torch.bincount(lab, minlength=k)
    C = torch.zeros((k, X.shape[1]), dtype=torch.float64, device="cuda")
    C.index_add_(0, lab, X)
    return C / cnt.clamp(min=1)[:, None], cnt


def _fit64(case, X, C):
    k, x2 = case["k"], float((X * X).sum())
    dead = torch.zeros(k, dtype=torch.bool, device="cuda") if case["empty"] == "exclude" else None
    it, last, obj = 0, 0.0, 0.0
    while it < case["maxiter"]:
        it += 1
        lab, best = _assign64(X, C, dead)
        obj = float(best.sum())
        new, cnt = _means64(X, lab, k)
        if dead is not None:
            dead = cnt == 0
        moved = float(((new - C) ** 2).sum(1).max().sqrt())
        C = new
        if case["conv"] == "shift" and it > 1 and moved <= case["tol"]:
            break
        if case["conv"] == "score":
            if it > 1 and abs(obj - x2 - last) < case["tol"]:
                break
            last = obj - x2
    return C, obj


def _kernel64(case, x, y):
    a = _kernel_args(case)
    if case["kernel"] == "gaussian":
        d2 = ((x * x).sum(1)[:, None] + (y * y).sum(1)[None, :]).addmm_(x, y.T, alpha=-2.0).clamp_(min=0)
        return d2.mul_(-1.0 / (2.0 * a["sigma"] ** 2)).exp_()
    dot = x @ y.T
    if case["kernel"] == "linear":
        return dot
    dot = dot.mul_(a["gamma"]).add_(a["coef"])
    return dot.square_() if case["kernel"] == "polynomial" else dot.tanh_()


def exact(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    if kind == "fit":
        # sample picks come from the framework's own seeded draws; the largest
        # fits take too long in 64 bits
        if case["init"] == "sample" or case["n"] * case["d"] * case["k"] * case["maxiter"] > 3e12:
            return None
        X, _ = _points(case, g)
        k = case["k"]
        if case["init"] == "given":
            C = _picked_rows(X, k, seed).double()
            X = X.double()
        else:
            X = X.double()
            C, _ = _means64(X, torch.arange(case["n"], device="cuda") % k, k)
        C, obj = _fit64(case, X, C)
        return {"labels": None, "centroids": C, "iterations": None, "converged_iter": None, "objective": obj}
    if kind == "assign":
        X, _ = _points(case, g)
        C = (_picked_rows(X, case["k"], seed) * 0.9).double()
        return {"labels": None, "mindist": _assign64(X.double(), C, None)[1]}
    if kind == "update":
        X, lab = _points(case, g)
        return {"centroids": _means64(X.double(), lab, case["k"])[0], "counts": None, "perm": None, "offsets": None}
    if kind == "kernel_matrix":
        X = _kernel_points(case, g).double()
        K = _kernel64(case, X, X)
        return {"K": K, "diag": K.diagonal().clone()}
    if kind == "kernel_fit":
        n, k = case["n"], case["k"]
        X = _kernel_points(case, g).double()
        K = torch.empty((n, n), dtype=torch.float64, device="cuda")
        for a in range(0, n, 4096):
            K[a:a + 4096] = _kernel64(case, X[a:a + 4096], X)
        lab = torch.arange(n, device="cuda") % k
        it, last, score = 0, 0.0, 0.0
        while it < case["maxiter"]:
            it += 1
            V = torch.nn.functional.one_hot(lab, k).double()
            E = K @ V
            cnt = V.sum(0)
            ct = (E * V).sum(0) / (cnt * cnt).clamp(min=1)
            D = E * (-2.0 / cnt.clamp(min=1))[None, :] + torch.where(ct == 0, math.inf, ct)[None, :]
            m, lab = D.min(1)
            score = float(m.sum())
            if case["check"] and 1 < it < case["maxiter"] and abs(score - last) < 1e-4:
                break
            last = score
        return {"labels": None, "iterations": None, "score": score}
    return None      # k-means++ and batched picks come from the framework's own seeded draws
