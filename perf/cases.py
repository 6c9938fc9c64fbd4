"""The workloads whose speed is measured: what a program that uses this library has it do.

Every case goes through the public entry points: the resident handle (kmgb_create ... kmgb_run),
the one-shot call, the drop-in drivers computeKmeansF/D on host arrays, the batched call, the
k-means++ draws and the reference's per-kernel entries on device arrays. Sizes are those of the
benchmark configurations, of the reference's own test matrices (898,790 x 128 with values of bytes
and 796,160 x 324 with values in [0, 1], K=256) and of this repository's tests.

A case is a dict of plain values:
  kind     handle | oneshot | driver | batched | kmeanspp | kernels
  n, d, k  rows, dimensions, centers (batched: `count` problems, their sizes drawn from `sizes`)
  values   blobs (Gaussian mixture, per-dimension std in [lo, hi], means U[-span, span]) | bytes
           (non-negative integers up to 255) | unit (values in [0, 1]) | zipf (many isotropic
           Gaussians of Zipf sizes, values that are BF16 numbers)
  iters    Lloyd iterations; tier: assignment tier; window: mini-batch fraction; dtype: f32 | f64
"""
import ctypes
import math

import numpy as np
import torch

import kmeans_gb300 as km

TIERS = {"fp32": km.ASSIGN_FP32, "bf16": km.ASSIGN_BF16, "split": km.ASSIGN_BF16X3,
         "auto": km.ASSIGN_AUTO}


def listed():
    return [
        # the smallest call in ordinary use: a notebook-sized data set in one call, host to host
        dict(name="oneshot_6k_x32_k16", kind="oneshot", n=6000, d=32, k=16, iters=10, tier="fp32",
             values="blobs", comps=16, span=10.0, lo=1.0, hi=1.0),
        # the benchmark's small configuration, resident: an iteration is many short kernels
        dict(name="handle_100k_x32_k64", kind="handle", n=100_000, d=32, k=64, iters=20,
             tier="split", window=1.0, values="blobs", comps=64, span=10.0, lo=1.0, hi=1.0),
        # the benchmark's headline configuration, resident
        dict(name="handle_4m_x128_k1024", kind="handle", n=4_000_000, d=128, k=1024, iters=10,
             tier="split", window=1.0, values="blobs", comps=1024, span=20.0, lo=0.3, hi=3.0),
        # rows wider than the tensor-core tier takes: the plain FP32 tier (the reference's HOG test)
        dict(name="handle_796k_x324_k256_fp32", kind="handle", n=796_160, d=324, k=256, iters=10,
             tier="fp32", window=1.0, values="unit", comps=256, span=1.0, lo=0.1, hi=0.1),
        # a large vocabulary: many centers against Zipf-sized clusters of BF16 numbers
        dict(name="handle_1m_x256_k16384", kind="handle", n=1_000_000, d=256, k=16384, iters=3,
             tier="split", window=1.0, values="zipf", comps=16384, span=5.0, lo=1.0, hi=1.0),
        # sliding mini-batch windows over a resident data set
        dict(name="handle_898k_x128_k256_window", kind="handle", n=898_790, d=128, k=256, iters=20,
             tier="split", window=0.1, values="bytes", comps=256, span=60.0, lo=30.0, hi=30.0),
        # the reference's own SIFT test through its driver entry, host to host
        dict(name="driver_f_898k_x128_k256", kind="driver", dtype="f32", n=898_790, d=128, k=256,
             iters=50, window=1.0, values="bytes", comps=256, span=60.0, lo=30.0, hi=30.0),
        # the double-precision driver
        dict(name="driver_d_400k_x64_k256", kind="driver", dtype="f64", n=400_000, d=64, k=256,
             iters=20, window=1.0, values="blobs", comps=256, span=4.0, lo=0.5, hi=2.0),
        # many independent problems in one call
        dict(name="batched_200", kind="batched", count=200, nmin=256, nmax=200_000, iters=15,
             tier="auto", sizes=2024),
        # k-means++ centers of a resident data set
        dict(name="kmeanspp_1m_x128_k256", kind="kmeanspp", n=1_000_000, d=128, k=256,
             dtype="f32", values="blobs", comps=256, span=20.0, lo=0.3, hi=3.0),
        # the reference's loop made of its per-kernel entries on device arrays, single precision
        dict(name="kernels_f_898k_x128_k256", kind="kernels", dtype="f32", n=898_790, d=128, k=256,
             iters=3, values="bytes", comps=256, span=60.0, lo=30.0, hi=30.0),
        # the same in double precision
        dict(name="kernels_d_100k_x64_k256", kind="kernels", dtype="f64", n=100_000, d=64, k=256,
             iters=3, values="blobs", comps=256, span=4.0, lo=0.5, hi=2.0),
    ]


# -------------------------------------------------------------------------------------------
# drawn cases
# -------------------------------------------------------------------------------------------

def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _values(rng, k):
    v = rng.choice(["blobs", "blobs", "bytes", "unit", "zipf"])
    if v == "blobs":
        lo = rng.uniform(0.3, 1.5)
        return dict(values=v, comps=max(1, _log(rng, max(1, k // 2), 2 * k)),
                    span=round(rng.uniform(2.0, 20.0), 3), lo=round(lo, 3),
                    hi=round(lo * rng.uniform(1.0, 4.0), 3))
    if v == "bytes":
        return dict(values=v, comps=k, span=60.0, lo=30.0, hi=30.0)
    if v == "zipf":
        return dict(values=v, comps=k, span=5.0, lo=1.0, hi=1.0)
    return dict(values=v, comps=k, span=1.0, lo=0.1, hi=0.1)


def _fit(n, per_row, most):
    """n, or fewer rows where n of them would cost more than `most`."""
    return max(64, min(n, int(most / per_row)))


def draw(rng):
    kind = rng.choice(["oneshot", "handle", "handle", "handle", "driver", "driver", "batched",
                       "kmeanspp", "kernels", "kernels"])
    if kind == "batched":
        return dict(kind=kind, count=_log(rng, 20, 200), nmin=256, nmax=_log(rng, 4000, 200_000),
                    iters=rng.randint(5, 15), tier=rng.choice(["auto", "split", "fp32"]),
                    sizes=rng.randint(1, 1 << 20))
    if kind == "kmeanspp":
        n, d, k = _log(rng, 2000, 2_000_000), _log(rng, 4, 256), _log(rng, 8, 256)
        dtype = rng.choice(["f32", "f32", "f64"])
        n = max(k, _fit(n, d * k, 3.2e10 if dtype == "f32" else 4e9))
        return dict(kind=kind, n=n, d=d, k=k, dtype=dtype, **_values(rng, k))
    if kind == "oneshot":
        n, d, k = _log(rng, 1000, 200_000), _log(rng, 2, 128), _log(rng, 2, 256)
        return dict(kind=kind, n=max(n, 4 * k), d=d, k=k, iters=rng.randint(3, 20),
                    tier=rng.choice(["fp32", "split"]), **_values(rng, k))
    if kind == "handle":
        tier = rng.choice(["split", "split", "split", "fp32", "bf16"])
        n, d = _log(rng, 4000, 4_000_000), _log(rng, 4, 320 if tier == "split" else 512)
        k = min(_log(rng, 8, 4096), n // 16)
        iters = rng.randint(3, 20)
        n = _fit(n, d * max(k, 64) * iters, 2e12 if tier == "split" else 2e11)
        k = min(k, max(2, n // 16))
        return dict(kind=kind, n=n, d=d, k=k, iters=iters, tier=tier,
                    window=rng.choice([1.0, 1.0, 1.0, 0.25]), **_values(rng, k))
    if kind == "driver":
        dtype = rng.choice(["f32", "f32", "f64"])
        n, d, k = _log(rng, 4000, 900_000), _log(rng, 4, 324), _log(rng, 8, 512)
        iters = rng.randint(5, 50)
        most = 4e11 if dtype == "f32" and d <= 320 else 1e11 if dtype == "f32" else 1e10
        n = _fit(n, d * max(k, 64) * iters, most)
        k = min(k, max(2, n // 16))
        return dict(kind=kind, dtype=dtype, n=n, d=d, k=k, iters=iters,
                    window=rng.choice([1.0, 1.0, 0.25]) if dtype == "f32" else 1.0,
                    **_values(rng, k))
    dtype = rng.choice(["f32", "f64"])
    n, d, k = _log(rng, 2000, 900_000), _log(rng, 4, 324), _log(rng, 8, 1024)
    iters = rng.randint(1, 4)
    n = _fit(n, d * max(k, 64) * iters, 1e11 if dtype == "f32" else 5e9)
    k = min(k, max(2, n // 16))
    return dict(kind=kind, dtype=dtype, n=n, d=d, k=k, iters=iters, **_values(rng, k))


# -------------------------------------------------------------------------------------------
# inputs
# -------------------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _data(case, g):
    """n x d float32 rows of the case's values, on the GPU."""
    n, d, comps = case["n"], case["d"], case["comps"]
    v, span = case["values"], case["span"]
    if v == "zipf":
        w = 1.0 / torch.arange(1, comps + 1, device="cuda", dtype=torch.float64) ** 1.1
        cdf = torch.cumsum(w / w.sum(), 0)
        u = torch.rand(n, device="cuda", generator=g, dtype=torch.float64)
        comp = torch.searchsorted(cdf, u).clamp_(max=comps - 1)
        means = torch.randn((comps, d), device="cuda", generator=g) * span
    else:
        comp = torch.randint(0, comps, (n,), device="cuda", generator=g)
        means = torch.empty((comps, d), device="cuda").uniform_(-span, span, generator=g)
        if v == "bytes":
            means += 20.0
        elif v == "unit":
            means = (means + 1.0) / 2.0
    if case["lo"] == case["hi"]:
        stds = torch.full((comps, d), float(case["lo"]), device="cuda")
    else:
        stds = torch.empty((comps, d), device="cuda").uniform_(
            math.log(case["lo"]), math.log(case["hi"]), generator=g).exp_()
    X = torch.empty((n, d), device="cuda")
    for s in range(0, n, 1 << 20):
        c = comp[s:s + (1 << 20)]
        X[s:s + (1 << 20)] = torch.randn((c.numel(), d), device="cuda", generator=g) * stds[c] + means[c]
    if v == "bytes":
        X.round_().clamp_(0.0, 255.0)
    elif v == "unit":
        X.clamp_(0.0, 1.0)
    elif v == "zipf":
        X = X.bfloat16().float()
    return X


def _wide(case, g):
    """The rows in the case's type; double-precision rows are not FP32 numbers."""
    X = _data(case, g)
    if case["dtype"] == "f64":
        X = X.double()
        if case["values"] != "bytes":
            X += 1e-9 * torch.rand(X.shape, device="cuda", generator=g, dtype=torch.float64)
    return X


def _init_rows(n, k, g):
    return torch.sort(torch.randperm(n, device="cuda", generator=g)[:k])[0]


def _sizes(case):
    """Sizes of the many-problems workload: rows log-uniform, D in {16, 32, 64, 128},
    K = sqrt(rows / 2) within [4, 512]."""
    rng = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["count"]):
        n = int(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]))))
        out.append((n, int(rng.choice([16, 32, 64, 128])),
                    int(min(512, max(4, round(math.sqrt(n / 2)))))))
    return out


def _problems(case, seed):
    g = _generator(seed)
    out = []
    for n, d, k in _sizes(case):
        means = torch.empty((k, d), device="cuda").uniform_(-10.0, 10.0, generator=g)
        comp = torch.randint(0, k, (n,), device="cuda", generator=g)
        X = torch.randn((n, d), device="cuda", generator=g) + means[comp]
        init = X[_init_rows(n, k, g)].cpu().numpy()
        out.append((X, k, init))
    return out


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case = case
    kind = case["kind"]
    if kind == "batched":
        st.problems = _problems(case, seed)
        torch.cuda.synchronize()
        return st
    g = _generator(seed)
    if kind in ("handle", "oneshot"):
        X = _data(case, g)
        init = X[_init_rows(case["n"], case["k"], g)].contiguous()
        if kind == "oneshot":
            st.X, st.init = X.cpu().numpy(), init.cpu().numpy()
        else:  # a program keeps the handle with its data set, and runs it from given centers
            st.init = init
            st.labels = torch.empty(case["n"], dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            st.handle = km.Handle(case["n"], case["d"], case["k"], assign_tier=TIERS[case["tier"]],
                                  empty_policy=km.EMPTY_KEEP, max_iters=case["iters"],
                                  mini_batch_fraction=case["window"])
            st.handle.set_data(X, on_device=True)
            st.handle.synchronize()
    elif kind == "driver":
        st.X = _wide(case, g).cpu().numpy()
        st.result = np.empty(case["k"] * case["d"], dtype=st.X.dtype)
    elif kind == "kmeanspp":
        st.X, st.seed = _wide(case, g), seed
    else:
        n, d, k = case["n"], case["d"], case["k"]
        t = torch.float32 if case["dtype"] == "f32" else torch.float64
        st.X = _wide(case, g)
        st.init = st.X[_init_rows(n, k, g)].contiguous()
        dev = dict(device="cuda")
        st.row_norms = torch.empty(n, dtype=t, **dev)
        st.col_norms = torch.empty(k, dtype=t, **dev)
        st.labels = torch.empty(n, dtype=torch.int32, **dev)
        st.centers = torch.empty((k, d), dtype=t, **dev)
        st.centers_large = torch.zeros(k * d, dtype=torch.float64, **dev)
        st.counts_large = torch.zeros(k, dtype=torch.int32, **dev)
        st.counts = torch.empty(k, dtype=torch.int32, **dev)
        st.compactness = torch.zeros(4, dtype=t, **dev)
    torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------------------------------
# one pass
# -------------------------------------------------------------------------------------------

def _ok(rc):
    if rc:
        raise RuntimeError("entry returned %d: %s" % (rc, km.last_error()))


def _run_handle(st):
    h, c = st.handle, st.case
    h.set_centers(st.init, on_device=True)
    h.run(c["iters"])
    h.synchronize()
    out = {"centers": h.centers(), "sse": h.sse(c["iters"])}
    if c["window"] >= 1.0:  # labels of the whole data set, into the caller's device array
        _ok(km.lib().kmgb_get_labels(h._h, ctypes.c_void_p(st.labels.data_ptr()), 1))
        out["labels"] = st.labels
    return out


def _run_kernels(st):
    """The reference's loop (norms, closest centers, cluster centers, transpose, compactness)."""
    c = st.case
    n, d, k = c["n"], c["d"], c["k"]
    if c["dtype"] == "f32":
        rownorm, colnorm, closest = km.rowNormalizeF, km.colNormalizeF, km.ClosestCentersF
        cluster, compact = km.ClusterCentersF, km.CompactnessF
    else:
        rownorm, colnorm, closest = km.rowNormalizeD, km.colNormalizeD, km.ClosestCentersD
        cluster, compact = km.ClusterCentersD, km.CompactnessD
    _ok(rownorm(0, n, d, st.X, st.row_norms))
    centers = st.init.t().contiguous()
    sse = []
    for _ in range(c["iters"]):
        st.centers_large.zero_()
        st.counts_large.zero_()
        st.compactness.zero_()
        _ok(colnorm(d, k, centers, st.col_norms))
        _ok(closest(0, n, d, st.X, k, centers, None, st.row_norms, st.col_norms, (k + 63) // 64,
                    None, None, st.labels))
        _ok(cluster(0, n, d, k, True, st.X, st.labels, st.centers_large, st.counts_large,
                    st.centers, st.counts))
        centers = st.centers.t().contiguous()
        _ok(compact(0, n, True, d, k, st.X, st.labels, st.centers, st.compactness))
        sse.append(st.compactness[0:1].clone())
    return {"row_norms": st.row_norms, "col_norms": st.col_norms, "centers": st.centers,
            "sse": torch.cat(sse), "labels": st.labels, "counts": st.counts}


def run(st):
    c = st.case
    kind = c["kind"]
    if kind == "handle":
        return _run_handle(st)
    if kind == "kernels":
        return _run_kernels(st)
    if kind == "oneshot":
        r = km.lloyd(st.X, c["k"], init=st.init, max_iters=c["iters"], assign_tier=TIERS[c["tier"]],
                     empty_policy=km.EMPTY_KEEP)
        return {"centers": r.centers, "sse": r.sse, "labels": r.labels}
    if kind == "driver":
        if c["dtype"] == "f32":
            rc = km.computeKmeansF(st.X, c["n"], c["d"], c["k"], -1.0, c["iters"], 1, 0, 0, 0,
                                   st.result, c["window"])
        else:
            rc = km.computeKmeansD(st.X, c["n"], c["d"], c["k"], -1.0, c["iters"], 1, 0, 0, 0,
                                   st.result, c["window"])
        if rc != km.KMEANS_NONCONVERGENCE:
            raise RuntimeError("driver returned %d: %s" % (rc, km.last_error()))
        return {"centers": st.result}
    if kind == "batched":
        res, _ = km.lloyd_batched(st.problems, max_iters=c["iters"], empty_policy=km.EMPTY_KEEP,
                                  assign_tier=TIERS[c["tier"]])
        return {"centers": np.concatenate([r.centers.ravel() for r in res]),
                "sse": np.concatenate([r.sse for r in res]),
                "labels": np.concatenate([r.labels for r in res])}
    centers, picks = km.kmeanspp(st.X, c["k"], seed=st.seed)
    return {"centers": centers, "picks": picks}


# -------------------------------------------------------------------------------------------
# what a pass cannot do without
# -------------------------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "batched":
        nb = fl = 0
        for n, d, k in _sizes(case):
            nb += case["iters"] * (4 * n * d + 8 * k * d) + 4 * n
            fl += case["iters"] * (2 * n * d * k + 3 * n * d)
        return {"bytes": nb, "flops": fl}
    n, d, k = case["n"], case["d"], case["k"]
    size = 8 if case.get("dtype") == "f64" else 4
    if kind == "kmeanspp":  # the rows once; per draw every row's squared distance read and written
        return {"bytes": size * n * d + 2 * size * n * k, "flops": 3 * n * d * k}
    m = int(case.get("window", 1.0) * n)
    per = size * (m * d + 2 * k * d) + 4 * m  # every iteration reads its rows, writes its labels
    fl = 2 * m * d * k + 3 * m * d
    if kind == "kernels":  # each entry reads the rows it is given
        return {"bytes": case["iters"] * (3 * size * n * d + 12 * n) + size * (n * d + n),
                "flops": case["iters"] * fl + 2 * n * d}
    once = size * n * d if kind in ("oneshot", "driver") else 0  # the upload
    return {"bytes": case["iters"] * per + once, "flops": case["iters"] * fl}


# -------------------------------------------------------------------------------------------
# the same in 64 bits
# -------------------------------------------------------------------------------------------

def _assign64(X, C, nb=None):
    """Arg-min over the rows of C (NaN rows never win): |x - c|^2, or nb - 2 x.c."""
    out = torch.empty(X.shape[0], dtype=torch.int64, device="cuda")
    if nb is None:
        nb = (C * C).sum(1)
    step = max(1, (1 << 28) // max(1, C.shape[0]))
    for s in range(0, X.shape[0], step):
        v = nb[None, :] - 2.0 * (X[s:s + step].double() @ C.t())
        out[s:s + step] = torch.nan_to_num(v, nan=math.inf).argmin(1)
    return out


def _means64(X, lab, old, keep):
    k, d = old.shape
    s = torch.zeros((k, d), dtype=torch.float64, device="cuda")
    step = 1 << 20
    for b in range(0, X.shape[0], step):
        s.index_add_(0, lab[b:b + step], X[b:b + step].double())
    cnt = torch.bincount(lab, minlength=k)
    mean = s / cnt[:, None].double()
    if keep:
        mean = torch.where(cnt[:, None] > 0, mean, old)
    return mean, cnt


def _sse64(X, lab, C):
    t = 0.0
    step = 1 << 20
    for b in range(0, X.shape[0], step):
        u = X[b:b + step].double() - C[lab[b:b + step]]
        t += float((u * u).sum())
    return t


def _lloyd64(X, init, iters, keep, f32, rows=None):
    """Lloyd's loop in 64 bits; the centers are numbers of the data's type between iterations.
    rows(t): the rows of iteration t (mini-batch windows)."""
    C = init.double()
    sse, lab = [], None
    for t in range(iters):
        Xi = X if rows is None else X[rows(t)]
        lab = _assign64(Xi, C)
        C, _ = _means64(Xi, lab, C, keep)
        if f32:
            C = C.float().double()
        sse.append(_sse64(Xi, lab, C))
    return C, np.array(sse), lab


def exact(case, seed):
    kind = case["kind"]
    if kind == "kmeanspp":  # the draws are of the data's rows: picks are whole numbers
        return None
    if kind == "batched":
        cen, sse = [], []
        if sum(n * d * k for n, d, k in _sizes(case)) * case["iters"] > 3e12:
            return None
        for X, k, init in _problems(case, seed):
            C, s, _ = _lloyd64(X, torch.from_numpy(init).cuda(), case["iters"], True, True)
            cen.append(C.cpu().numpy().ravel())
            sse.append(s)
        return {"centers": np.concatenate(cen), "sse": np.concatenate(sse), "labels": None}
    n, d, k, iters = case["n"], case["d"], case["k"], case["iters"]
    if n * d * k * iters > 6e12 or (kind == "driver" and case["window"] < 1.0):
        return None
    g = _generator(seed)
    if kind in ("handle", "oneshot"):
        X = _data(case, g)
        init = X[_init_rows(n, k, g)]
        if kind == "handle" and case["window"] < 1.0:  # the windows follow the library's shuffle
            return None
        C, sse, _ = _lloyd64(X, init, iters, True, True)
        return {"centers": C, "sse": sse, "labels": None}
    if kind == "driver":  # the initial rows come from the library's shuffle and picks
        return None
    X = _wide(case, g)
    f32 = case["dtype"] == "f32"
    C = X[_init_rows(n, k, g)].double()
    sse = []
    for _ in range(iters):
        nb = (C * C).sum(1)
        lab = _assign64(X, C, nb.float().double() if f32 else nb)
        C, cnt = _means64(X, lab, C, False)
        C = C.float().double() if f32 else C
        sse.append(_sse64(X, lab, C))
    return {"row_norms": torch.cat([(x.double() ** 2).sum(1) for x in X.split(1 << 20)]),
            "col_norms": nb, "centers": C, "sse": np.array(sse), "labels": None, "counts": None}
