"""The stop rule's criterion belongs to the run: a handle whose captured iteration is replayed by later
runs follows each run's own criterion."""
import numpy as np
import pytest

from kmeans_gb300.synthetic import mixture_numpy, sample_init

pytestmark = pytest.mark.gpu

N, D, K, ITERS, C = 20_000, 32, 24, 40, 1e-3


def data():
    X, _, _ = mixture_numpy(N, D, K, seed=5, mean_lo=-4, mean_hi=4, std=(1.0, 1.0))
    return X, X[sample_init(N, K, seed=6)].copy()


@pytest.mark.parametrize("tier", ["FP32", "BF16X3"])
@pytest.mark.parametrize("order", [(-1.0, C), (C, -1.0), (-1.0, C, -1.0, 10 * C)])
def test_each_run_follows_its_own_criterion(km, orc, torch_cuda, tier, order):
    X, init = data()
    h = km.Handle(N, D, K, assign_tier=getattr(km, "ASSIGN_" + tier), empty_policy=1, max_iters=ITERS)
    h.set_data(X, on_device=False)
    for c in order:
        st, cen, lab, sse, it = orc.lloyd(X, init, ITERS, criterion=c, empty_policy=1)
        assert (it < ITERS) == (c > 0)
        h.set_centers(init)
        h.run(ITERS, c)
        h.synchronize()
        s = h.stats()
        assert (s.iterations, s.status) == (it, st), c
        assert np.array_equal(h.centers(), cen) and np.array_equal(h.labels(), lab), c
    h.close()


@pytest.mark.parametrize("order", [(-1.0, 0.05), (0.05, -1.0)])
def test_windows_follow_their_runs_criterion(km, torch_cuda, monkeypatch, order):
    """Mini-batch windows move on from run to run, so the second run is checked against its own SSE
    history without a criterion and against the launches one by one."""
    X, init = data()

    def go(criteria, graphs):
        monkeypatch.setenv("KMGB_GRAPHS", graphs)
        h = km.Handle(N, D, K, assign_tier=km.ASSIGN_BF16X3, empty_policy=1, max_iters=ITERS,
                      mini_batch_fraction=0.2)
        h.set_data(X, on_device=False)
        h.set_centers(init)
        out = []
        for c in criteria:
            h.run(ITERS, c)
            h.synchronize()
            it = h.stats().iterations
            out.append((it, h.sse(it), h.centers()))
        h.close()
        return out

    free = go((order[0], -1.0), "0")[1][1]  # the second run's SSE where nothing stops it
    rel = np.abs(np.diff(free, prepend=0.0)) / np.abs(free)
    hit = np.nonzero(~(rel > order[1]))[0]
    want = int(hit[0]) + 1 if order[1] >= 0 and hit.size else ITERS
    assert (want < ITERS) == (order[1] > 0)
    a, b = go(order, "1"), go(order, "0")
    assert a[1][0] == b[1][0] == want
    for x, y in zip(a, b):
        assert np.array_equal(x[1], y[1]) and np.array_equal(x[2], y[2])
