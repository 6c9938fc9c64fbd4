"""Dimensions whose tiles need nearly all of the shared memory that a launch gets without asking for
more, each in a process that has launched nothing wider (which would have asked)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import numpy as np, torch, oracle
import kmeans_gb300 as km
oracle.build()
for d in %r:
    rng = np.random.default_rng(d)
    X = rng.integers(-20, 21, (400, d)).astype(np.float32)
    X[100:140] = X[100]
    init = X[rng.choice(100, 9, replace=False)].copy()
    init[3] = init[7] = X[100]
    want = oracle.lloyd(X, init, 2, empty_policy=1)
    for tier in (km.ASSIGN_FP32, km.ASSIGN_BF16X3):
        r = km.lloyd(X, 9, init=init, max_iters=2, assign_tier=tier, empty_policy=1)
        assert np.array_equal(r.labels, want[2]) and np.array_equal(r.centers, want[1]), d
    a, b = torch.from_numpy(X).cuda(), torch.from_numpy(np.ascontiguousarray(init.T)).cuda()
    nb = (b * b).sum(0)
    lab = torch.full((400,), -1, dtype=torch.int32, device="cuda")
    assert km.ClosestCentersF(0, 400, d, a, 9, b, None, None, nb, 0, None, None, lab) == 0, d
    v = nb.cpu().numpy().astype(float)[None] - 2.0 * X.astype(float) @ init.T.astype(float)
    assert np.array_equal(lab.cpu().numpy(), v.argmin(1)), d
print("ok")
"""


@pytest.mark.parametrize("dims", [(97, 100, 104), (105, 108, 112), (113, 116, 117, 120), (121, 124)])
def test_dimensions_near_the_plain_shared_memory_limit(torch_cuda, dims):
    r = subprocess.run([sys.executable, "-c", CODE % (dims,)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]
