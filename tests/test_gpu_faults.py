"""Failure paths, through the C-ABI, without faulting the GPU.

Host-side injection (kmgb_debug_fail_nth) makes one allocation, copy or kernel launch of a call
fail as the CUDA call would have failed: the call must return the kmeansErrorStatus of the phase
it was in (the reference reports failures only through these codes, kmeans.hpp:44-59), leave a
message, give back every byte it took from the library's memory pool, and leave the context usable
(the next call returns the oracle's result). A bounded device wait is made to run out by
withholding one TMA load of the FP32 assignment (kmgb_debug_withhold_stage) with a short wait
limit: every load issued before it has been consumed, so nothing is left in flight, and the kernel
reports the timeout through the device error word."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, D, K, ITERS = 5000, 24, 12, 3


@pytest.fixture()
def no_graphs():
    old = os.environ.get("KMGB_GRAPHS")
    os.environ["KMGB_GRAPHS"] = "0"  # kernel-by-kernel launches: the event order is fixed
    yield
    if old is None:
        os.environ.pop("KMGB_GRAPHS")
    else:
        os.environ["KMGB_GRAPHS"] = old


def data():
    from kmeans_gb300.synthetic import mixture_numpy, sample_init
    X, _, _ = mixture_numpy(N, D, K, seed=21)
    return X, X[sample_init(N, K, seed=22)].copy()


def call(km, X, init, tier):
    try:
        res = km.lloyd(X, K, init=init, max_iters=ITERS, assign_tier=tier)
        return 0, res
    except km.KmeansError as e:
        return e.code, None


def check_clean(km, torch, orc, X, init, tier, base_used):
    torch.cuda.synchronize()
    assert km.debug_pool_used_bytes() == base_used, "pool memory not given back"
    rc, res = call(km, X, init, tier)
    assert rc == 0
    st, c, lab, sse, it = orc.lloyd(X, init, ITERS)
    assert np.array_equal(res.labels, lab) and np.array_equal(res.centers, c)


@pytest.mark.parametrize("tier_name", ["fp32", "bf16x3"])
def test_injected_failures_return_phase_codes_and_release_memory(km, orc, torch_cuda, no_graphs,
                                                                  tier_name):
    torch = torch_cuda
    tier = {"fp32": km.ASSIGN_FP32, "bf16x3": km.ASSIGN_BF16X3}[tier_name]
    X, init = data()
    call(km, X, init, tier)  # warm: module loading, pool creation
    torch.cuda.synchronize()
    base = km.debug_pool_used_bytes()
    assert base >= 0
    valid = set(range(1, 13))
    seen = {}
    for kind in (km.FAULT_ALLOC, km.FAULT_COPY, km.FAULT_LAUNCH):
        nth = 1
        while True:
            km.debug_fail_nth(kind, nth)
            rc, res = call(km, X, init, tier)
            km.debug_fail_nth(kind, 0)
            if rc == 0:  # more events asked for than the call has: it ran untouched
                break
            assert rc in valid, (kind, nth, rc)
            assert km.last_error(), (kind, nth)
            seen[(kind, nth)] = rc
            check_clean(km, torch, orc, X, init, tier, base)
            nth += 1
            assert nth < 200
    # the first allocation is the handle's arena (KMEANS_ERROR_BUILDDATA); the second copy
    # uploads the initial centers (KMEANS_ERROR_INITIALIZE)
    assert seen[(km.FAULT_ALLOC, 1)] == km.KMEANS_ERROR_BUILDDATA
    assert seen[(km.FAULT_COPY, 2)] == km.KMEANS_ERROR_INITIALIZE
    codes = set(seen.values())
    # every phase of an iteration was reached by some launch failure: center preparation
    # (reset), assignment / re-rank (closest centers) and the update (cluster centers)
    assert {km.KMEANS_ERROR_RESET, km.KMEANS_ERROR_CLOSEST_CENTERS, km.KMEANS_ERROR_CLUSTER_CENTERS} <= {seen[k] for k in seen if k[0] == km.FAULT_LAUNCH}, seen
    assert codes <= valid


def test_withheld_tma_load_times_out_and_reports(km, orc, torch_cuda, no_graphs):
    torch = torch_cuda
    from kmeans_gb300.synthetic import mixture_numpy, sample_init
    # D = 100: four 32-float k-blocks per center chunk, so every CTA's pipeline has 4 steps
    X, _, _ = mixture_numpy(N, 100, K, seed=23)
    init = X[sample_init(N, K, seed=24)].copy()
    call(km, X, init, km.ASSIGN_FP32)
    torch.cuda.synchronize()
    base = km.debug_pool_used_bytes()
    # step 2 of every CTA's pipeline is never loaded; each wait gives up after 2e6 SM cycles
    # (about a millisecond)
    km.debug_withhold_stage(2, 2_000_000)
    try:
        rc, _ = call(km, X, init, km.ASSIGN_FP32)
    finally:
        km.debug_withhold_stage(0, 0)
    assert rc == km.KMEANS_ERROR_CLOSEST_CENTERS
    assert "device error word 1" in km.last_error()  # KMGB_DEV_TIMEOUT_FULL
    check_clean(km, torch, orc, X, init, km.ASSIGN_FP32, base)


def test_failure_inside_graph_capture_falls_back(km, orc, torch_cuda):
    """With graphs on, a launch failure injected while the iteration is being captured aborts
    the capture; the run then launches kernel by kernel and returns the oracle's result."""
    X, init = data()
    call(km, X, init, km.ASSIGN_FP32)
    # the launches of one-time work come first (norms); the capture starts with the first
    # iteration's center preparation
    km.debug_fail_nth(km.FAULT_LAUNCH, 2)
    try:
        rc, res = call(km, X, init, km.ASSIGN_FP32)
    finally:
        km.debug_fail_nth(km.FAULT_LAUNCH, 0)
    assert rc == 0
    st, c, lab, sse, it = orc.lloyd(X, init, ITERS)
    assert np.array_equal(res.labels, lab) and np.array_equal(res.centers, c)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_closest_centers_without_room_for_its_planes(km, torch_cuda, dtype):
    """Sizes that take the tensor-core filter: where its workspace does not fit, the scans that
    need less memory (FP64: none) give the same labels."""
    torch = torch_cuda
    rng = np.random.default_rng(8)
    n, d, k = 60_000, 64, 128
    A = (rng.integers(-40, 41, (n, d)) / 8).astype(dtype)
    B = (rng.integers(-40, 41, (d, k)) / 8).astype(dtype)
    nb = (B.astype(np.float64) ** 2).sum(0).astype(dtype)
    want = (nb.astype(np.float64)[None] - 2.0 * (A.astype(np.float64) @ B.astype(np.float64))).argmin(1)
    a, b, c = (torch.from_numpy(v).cuda() for v in (A, B, nb))
    fn = km.ClosestCentersF if dtype == np.float32 else km.ClosestCentersD
    for nth in (0, 1):
        out = torch.full((n,), -7, dtype=torch.int32, device="cuda")
        km.debug_fail_nth(km.FAULT_ALLOC, nth)
        try:
            assert fn(0, n, d, a, k, b, None, None, c, 0, None, None, out) == 0
        finally:
            km.debug_fail_nth(km.FAULT_ALLOC, 0)
        assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("kpp", [False, True])
def test_double_precision_driver_without_its_optional_memory(km, torch_cuda, kpp):
    """The candidates' buffers may be smaller, the bounds' and the draws' row-skipping arrays missing:
    an allocation that fails among them leaves the result as it is; among the others the call fails
    and gives everything back."""
    rng = np.random.default_rng(4)
    n, d, k = 140_000, 64, 200
    means = rng.uniform(-4, 4, (k, d))
    X = means[rng.integers(0, k, n)] + rng.standard_normal((n, d))

    def go():
        out = np.empty(k * d)
        return km.computeKmeansD(X, n, d, k, -1.0, 4, 1, km.INIT_KMEANSPP if kpp else 0, 0, 0, out, 1.0), out

    rc, want = go()
    assert rc == km.KMEANS_NONCONVERGENCE
    base = km.debug_pool_used_bytes()
    failed = 0
    for nth in range(1, 61):  # the call makes some fifty allocations
        km.debug_fail_nth(km.FAULT_ALLOC, nth)
        rc, got = go()
        km.debug_fail_nth(km.FAULT_ALLOC, 0)
        torch_cuda.cuda.synchronize()
        assert km.debug_pool_used_bytes() == base
        if rc == km.KMEANS_NONCONVERGENCE:
            assert np.array_equal(got, want, equal_nan=True)  # (an empty cluster is NaN)
        else:
            assert rc in range(1, 13)
            failed += 1
    # the required buffers alone: not the five of the candidates, the fifteen of the bounds and the
    # draws' two
    assert 0 < failed <= (37 if kpp else 32)


@pytest.mark.parametrize("d", [24, 64])
def test_fp32_handle_without_room_for_its_extras(km, orc, torch_cuda, d):
    """The FP32 tier's transposed centers and band candidates are left out where they do not fit:
    same labels and centers (d = 64: with distance bounds)."""
    from kmeans_gb300.synthetic import mixture_numpy, sample_init
    n, k = 70_000, 40
    X, _, _ = mixture_numpy(n, d, k, seed=31)
    X[50:60] = X[50]
    init = X[sample_init(n, k, seed=32)].copy()
    init[3] = init[9] = X[50]
    want = orc.lloyd(X, init, 5, empty_policy=1)
    km.debug_fail_nth(km.FAULT_ALLOC, 1)
    try:
        res = km.lloyd(X, k, init=init, max_iters=5, assign_tier=km.ASSIGN_FP32, empty_policy=1)
    finally:
        km.debug_fail_nth(km.FAULT_ALLOC, 0)
    assert np.array_equal(res.labels, want[2]) and np.array_equal(res.centers, want[1])


@pytest.mark.parametrize("dtype,n", [(np.float32, 5_000), (np.float32, 60_000), (np.float64, 60_000)])
def test_closest_centers_after_a_wait_that_gave_up(km, torch_cuda, dtype, n):
    """The entry returns before its kernels have run: where a bounded wait of the scan gives up, its
    last kernel settles every row. (60,000 rows take the tensor-core filter, whose given-up wait is
    stood in for by its error word and labels of -1.)"""
    torch = torch_cuda
    rng = np.random.default_rng(9)
    d, k = 100, 128
    A = (rng.integers(-40, 41, (n, d)) / 8).astype(dtype)
    B = (rng.integers(-40, 41, (d, k)) / 8).astype(dtype)
    nb = (B.astype(np.float64) ** 2).sum(0).astype(dtype)
    want = (nb.astype(np.float64)[None] - 2.0 * (A.astype(np.float64) @ B.astype(np.float64))).argmin(1)
    a, b, c = (torch.from_numpy(v).cuda() for v in (A, B, nb))
    fn = km.ClosestCentersF if dtype == np.float32 else km.ClosestCentersD
    out = torch.full((n + 2,), -7, dtype=torch.int32, device="cuda")
    km.debug_withhold_stage(2, 2_000_000)
    try:
        assert fn(2, n, d, a, k, b, None, None, c, 0, None, None, out) == 0
        torch.cuda.synchronize()
    finally:
        km.debug_withhold_stage(0, 0)
    assert np.array_equal(out.cpu().numpy()[2:], want)


def test_batched_upload_with_less_pinned_memory(km, orc, torch_cuda, no_graphs):
    """Page-locked staging that cannot be had at its size is taken smaller: among the allocations of a
    call made to fail in turn, its two leave the result as it is; the ones before and after fail the
    call."""
    from kmeans_gb300.synthetic import mixture_numpy, sample_init
    probs = []
    for i, (n, d, k) in enumerate([(9000, 24, 8), (7001, 24, 5), (20_000, 24, 12)]):
        X, _, _ = mixture_numpy(n, d, k, seed=80 + i)
        probs.append((X, k, X[sample_init(n, k, seed=i)].copy()))
    want = [orc.lloyd(X, init, 3) for X, _, init in probs]
    ran = []
    for nth in range(1, 81):
        km.debug_fail_nth(km.FAULT_ALLOC, nth)
        try:
            res, _ = km.lloyd_batched(probs, max_iters=3, assign_tier=km.ASSIGN_FP32)
            ran.append(True)
            for r, w in zip(res, want):
                assert np.array_equal(r.labels, w[2]) and np.array_equal(r.centers, w[1])
        except km.KmeansError:
            ran.append(False)
        finally:
            km.debug_fail_nth(km.FAULT_ALLOC, 0)
    first = ran.index(True)
    assert first > 0 and ran[first:first + 3] == [True, True, False]
    assert ran[-1]  # past the call's last allocation
