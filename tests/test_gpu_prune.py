"""Distance bounds kept between the iterations of a run: runs large enough to use them (rows x
centers x dimensions at or above the handle's threshold) must equal the oracle's loop bit for bit
in labels and centers, whatever share of the rows an iteration scans."""
import numpy as np
import pytest

from kmeans_gb300.synthetic import mixture_numpy, sample_init

pytestmark = pytest.mark.gpu


def check(res, want, name=""):
    st, c, lab, sse, it = want
    assert res.iterations == it and res.status == st, name
    assert np.array_equal(res.labels, lab), f"{name}: labels"
    assert np.array_equal(res.centers, c, equal_nan=True), f"{name}: centers"
    np.testing.assert_allclose(res.sse, sse, rtol=1e-10)
    assert res.audit_violations == 0


CASES = [
    # n, d, k, components, mean span, std, tier, BF16-valued, policy
    (70_001, 128, 1000, 1000, 20.0, (0.3, 3.0), "BF16X3", False, 1),  # separated: most rows skipped
    (66_003, 129, 1024, 64, 2.0, (1.0, 1.0), "BF16X3", False, 1),     # overlapping: most rows scanned
    (140_000, 256, 256, 200, 8.0, (0.5, 1.5), "BF16X3", True, 0),     # two products, NaN policy
    (132_777, 130, 500, 500, 20.0, (1.0, 1.0), "BF16", False, 1),     # plain tier
    (90_001, 324, 300, 300, 1.0, (0.1, 0.1), "FP32", False, 1),       # FP32 tier, wide rows
    (100_003, 45, 700, 80, 2.0, (1.0, 1.0), "FP32", False, 0),
    (600_000, 60, 250, 240, 10.0, (1.0, 1.0), "BF16X3", False, 1),
]


@pytest.mark.parametrize("n,d,k,comps,span,std,tier,bf16,policy", CASES)
def test_bounds_match_oracle(km, orc, torch_cuda, n, d, k, comps, span, std, tier, bf16, policy):
    X, _, _ = mixture_numpy(n, d, comps, seed=n, mean_lo=-span, mean_hi=span, std=std)
    if bf16:
        X = torch_cuda.from_numpy(X).bfloat16().float().numpy()
    X[100:140] = X[100]  # duplicate rows: exact ties between duplicate centers
    init = X[sample_init(n, k, seed=3)].copy()
    init[7] = init[2] = X[100]
    want = orc.lloyd(X, init, 8, empty_policy=policy)
    t = getattr(km, "ASSIGN_" + tier)
    # host rows travel with the first iteration, device rows do not
    check(km.lloyd(X, k, init=init, max_iters=8, assign_tier=t, empty_policy=policy), want, "host")
    Xd = torch_cuda.from_numpy(X).cuda()
    check(km.lloyd(Xd, k, init=init, max_iters=8, assign_tier=t, empty_policy=policy), want, "device")


def test_bounds_end_with_the_run(km, orc, torch_cuda, monkeypatch):
    """Other centers, other data and single-iteration runs on one handle start without bounds; a
    run that converges stops in the oracle's iteration; kernel-by-kernel launches agree."""
    n, d, k = 70_001, 128, 1000
    X, _, _ = mixture_numpy(n, d, k, seed=11, mean_lo=-20, mean_hi=20, std=(0.3, 3.0))
    Y, _, _ = mixture_numpy(n, d, k, seed=12, mean_lo=-20, mean_hi=20, std=(0.3, 3.0))
    i1, i2 = X[sample_init(n, k, seed=1)], X[sample_init(n, k, seed=2)]
    h = km.Handle(n, d, k, assign_tier=km.ASSIGN_BF16X3, empty_policy=1, max_iters=6)

    def run(init, data, iters):
        if init is not None:
            h.set_centers(init)
        h.run(iters)
        h.synchronize()
        return h.labels(), h.centers()

    h.set_data(X, on_device=False)
    for init in (i1, i2):
        _, c, lab, _, _ = orc.lloyd(X, init, 5, empty_policy=1)
        got = run(init, X, 5)
        assert np.array_equal(got[0], lab) and np.array_equal(got[1], c)
    _, c, lab, _, _ = orc.lloyd(X, c, 1, empty_policy=1)
    got = run(None, X, 1)  # continues from its centers
    assert np.array_equal(got[0], lab) and np.array_equal(got[1], c)
    h.set_data(Y, on_device=False)
    _, c, lab, _, _ = orc.lloyd(Y, i2, 4, empty_policy=1)
    got = run(i2, Y, 4)
    assert np.array_equal(got[0], lab) and np.array_equal(got[1], c)
    h.close()
    want = orc.lloyd(X, i1, 40, criterion=1e-3, empty_policy=1)
    for graphs in ("1", "0"):
        monkeypatch.setenv("KMGB_GRAPHS", graphs)
        check(km.lloyd(X, k, init=i1, max_iters=40, criterion=1e-3, empty_policy=1,
                       assign_tier=km.ASSIGN_BF16X3), want, "criterion")


@pytest.mark.parametrize("n,d,k,span", [(70_001, 128, 250, 20.0), (150_000, 66, 256, 2.0)])
def test_fp64_driver(km, orc, torch_cuda, n, d, k, span):
    """computeKmeansD with bounds: FP64-only digits in the rows, exact duplicates."""
    X, _, _ = mixture_numpy(n, d, k, seed=n, mean_lo=-span, mean_hi=span, std=(0.5, 2.0))
    X = X.astype(np.float64) + np.random.default_rng(1).uniform(0, 1e-9, X.shape)
    X[50:90] = X[50]
    _, perm, picks = km.reference_init(X.astype(np.float32), k)
    init = X[perm[picks]]
    result = np.empty(k * d)
    assert km.computeKmeansD(X, n, d, k, -1.0, 6, 1, 0, 0, 0, result, 1.0) == 13
    _, c, _, _, _ = orc.lloyd_d(X, init, 6)
    assert np.array_equal(result.reshape(d, k).T, c, equal_nan=True)


def large():
    n, d, k = 70_001, 128, 1000
    X, _, _ = mixture_numpy(n, d, k, seed=31, mean_lo=-20, mean_hi=20, std=(0.3, 3.0))
    return n, d, k, X, X[sample_init(n, k, seed=5)].copy()


def test_bounds_memory_only_where_it_is_used(km, orc, torch_cuda, monkeypatch):
    """A handle for single iterations and a sharded one hold what a handle without bounds holds; a
    longer run takes the memory when it comes."""
    n, d, k, X, init = large()
    torch_cuda.cuda.synchronize()
    base = km.debug_pool_used_bytes()

    def held(h):
        h.synchronize()
        torch_cuda.cuda.synchronize()
        return km.debug_pool_used_bytes() - base

    def make(max_iters):
        h = km.Handle(n, d, k, assign_tier=km.ASSIGN_BF16X3, empty_policy=1, max_iters=max_iters)
        h.set_data(X, on_device=False)
        h.set_centers(init)
        return h

    monkeypatch.setenv("KMGB_BOUNDS", "0")
    plain = make(6)
    least = held(plain)
    S0, c0, Q0 = plain.shard_partials()
    least_shard = held(plain)
    plain.close()
    monkeypatch.delenv("KMGB_BOUNDS")

    h = make(6)
    assert held(h) > least + n * 20
    S, c, Q = h.shard_partials()
    assert held(h) == least_shard
    assert np.array_equal(S, S0) and np.array_equal(c, c0) and np.array_equal(Q, Q0)
    h.shard_update(S, c, Q)
    one = orc.lloyd_tiled(X, init, 1, tile_rows=n, empty_policy=1)
    assert np.array_equal(h.centers(), one[1])
    h.close()

    h = make(1)
    h.run(1)
    assert held(h) <= least
    h.set_centers(init)
    h.run(5)  # after a captured iteration without bounds
    h.synchronize()
    want = orc.lloyd(X, init, 5, empty_policy=1)
    assert np.array_equal(h.centers(), want[1]) and np.array_equal(h.labels(), want[2])
    assert held(h) > least + n * 20
    h.close()
    assert km.debug_pool_used_bytes() == base


def test_bounds_give_way_to_memory_a_call_needs(km, orc, torch_cuda):
    n, d, k, X, init = large()
    h = km.Handle(n, d, k, assign_tier=km.ASSIGN_BF16X3, empty_policy=1, max_iters=4)
    h.set_data(X, on_device=False)
    h.set_centers(init)
    h.run(2)
    h.synchronize()
    km.debug_fail_nth(km.FAULT_ALLOC, 1)
    try:
        picks = h.init_kmeanspp(3)
    finally:
        km.debug_fail_nth(km.FAULT_ALLOC, 0)
    assert len(set(picks.tolist())) == k
    h.set_centers(init)
    h.run(4)
    h.synchronize()
    want = orc.lloyd(X, init, 4, empty_policy=1)
    assert np.array_equal(h.centers(), want[1]) and np.array_equal(h.labels(), want[2])
    h.close()


def test_bounds_without_room(km, orc, torch_cuda):
    """The bounds' own allocation (the third of a call) does not fit: every row is scanned."""
    n, d, k, X, init = large()
    km.debug_fail_nth(km.FAULT_ALLOC, 3)
    try:
        res = km.lloyd(X, k, init=init, max_iters=5, assign_tier=km.ASSIGN_BF16X3, empty_policy=1)
    finally:
        km.debug_fail_nth(km.FAULT_ALLOC, 0)
    check(res, orc.lloyd(X, init, 5, empty_policy=1))


@pytest.mark.parametrize("tier", ["BF16X3", "FP32"])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e30])
def test_bounds_with_rows_that_spoil_a_center(km, torch_cuda, monkeypatch, tier, value):
    n, d, k, X, init = large()
    X[5, 3] = X[60_000, 100] = value
    t = getattr(km, "ASSIGN_" + tier)
    got = km.lloyd(X, k, init=init, max_iters=5, assign_tier=t, empty_policy=1)
    monkeypatch.setenv("KMGB_BOUNDS", "0")
    want = km.lloyd(X, k, init=init, max_iters=5, assign_tier=t, empty_policy=1)
    assert np.array_equal(got.labels, want.labels)
    assert np.array_equal(got.centers, want.centers, equal_nan=True)


@pytest.mark.parametrize("graphs", ["1", "0"])
def test_run_length_decides(km, orc, torch_cuda, monkeypatch, graphs):
    """Short and long runs of one handle in turn (without and with bounds, each its own capture), and a
    handle created for short runs that gets a long one."""
    monkeypatch.setenv("KMGB_GRAPHS", graphs)
    n, d, k, X, init = large()
    want = {it: orc.lloyd(X, init, it, empty_policy=1) for it in (1, 3, 4, 6)}
    for max_iters, runs in ((8, (3, 6, 1, 4)), (2, (1, 3, 6, 3))):
        h = km.Handle(n, d, k, assign_tier=km.ASSIGN_BF16X3, empty_policy=1, max_iters=max_iters)
        h.set_data(X, on_device=False)
        for it in runs:
            h.set_centers(init)
            h.run(it)
            h.synchronize()
            assert np.array_equal(h.centers(), want[it][1]) and np.array_equal(h.labels(), want[it][2])
        h.close()


@pytest.mark.parametrize("tier", ["BF16X3", "FP32"])
@pytest.mark.parametrize("device", [False, True])
def test_bounds_after_tests_that_listed_too_many_rows(km, orc, torch_cuda, tier, device):
    """Byte-valued rows whose first tests fail (so that the next iterations go untested) and whose later
    ones hold: every iteration's state is that of the oracle's loop."""
    n, d, k = 70_000, 128, 256
    rng = np.random.default_rng(17)
    means = rng.uniform(-60, 60, (k, d)) + 20
    X = np.clip(np.round(means[rng.integers(0, k, n)] + 30 * rng.standard_normal((n, d))), 0, 255)
    X = X.astype(np.float32)
    init = X[sample_init(n, k, seed=18)].copy()
    src = torch_cuda.from_numpy(X).cuda() if device else X
    for iters in (5, 9, 24):
        check(km.lloyd(src, k, init=init, max_iters=iters, assign_tier=getattr(km, "ASSIGN_" + tier),
                       empty_policy=1), orc.lloyd(X, init, iters, empty_policy=1), iters)
