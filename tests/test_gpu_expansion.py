"""ClosestCentersF/D on the tensor-core filter, CompactnessF/D and the norms at the sizes where their
paths change: labels equal the FP64 evaluation of nb_j - 2 a.b_j (lowest index on ties) whatever
the norms, the sums FP64's within the FP32 rounding of the outputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact_labels(A, B, nb):
    A, B, nb = (np.asarray(v, np.float64) for v in (A, B, nb))
    out = np.empty(len(A), np.int32)
    for s in range(0, len(A), 4096):
        acc = np.zeros((len(A[s:s + 4096]), B.shape[1]))
        for t in range(B.shape[0]):  # the entry's order: one chain over the dimensions
            acc += A[s:s + 4096, t, None] * B[None, t]
        v = nb[None] - 2.0 * acc
        v[np.isnan(v)] = np.inf
        out[s:s + 4096] = v.argmin(1)
    return out


def closest(km, torch, A, B, nb, m0=3):
    dev = "cuda"
    F = A.dtype == np.float32
    a, b, n = (torch.from_numpy(np.ascontiguousarray(v)).to(dev) for v in (A, B, nb))
    out = torch.full((len(A) + m0,), -7, dtype=torch.int32, device=dev)
    fn = km.ClosestCentersF if F else km.ClosestCentersD
    assert fn(m0, A.shape[0], A.shape[1], a, B.shape[1], b, None, None, n, 0, None, None, out) == 0
    got = out.cpu().numpy()
    assert (got[:m0] == -7).all()
    return got[m0:]


# values on a grid of 1/8: every product and sum is exact in FP64, so equal values are exact ties
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,d,k", [(20_000, 128, 256), (40_001, 33, 300), (9_000, 320, 129),
                                   (30_000, 321, 64), (600_000, 7, 65), (70_000, 5, 3)])
def test_closest_centers_grid(km, torch_cuda, dtype, n, d, k):
    rng = np.random.default_rng(n + d + k)
    A = (rng.integers(-40, 41, (n, d)) / 8).astype(dtype)
    B = (rng.integers(-40, 41, (d, k)) / 8).astype(dtype)
    B[:, k - 1] = B[:, 0]  # duplicate centers: the lower index wins
    nb = (B.astype(np.float64) ** 2).sum(0).astype(dtype)
    A[:k] = B.T[: min(k, n)]
    assert np.array_equal(closest(km, torch_cuda, A, B, nb), exact_labels(A, B, nb))


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("case", ["nan center", "inf norm", "minus inf norm", "zero norms",
                                  "huge center", "inf row", "nan row", "all equal"])
def test_closest_centers_special(km, torch_cuda, dtype, case):
    rng = np.random.default_rng(5)
    n, d, k = 20_000, 64, 256
    A = (rng.integers(-40, 41, (n, d)) / 8).astype(dtype)
    B = (rng.integers(-40, 41, (d, k)) / 8).astype(dtype)
    nb = (B.astype(np.float64) ** 2).sum(0).astype(dtype)
    if case == "nan center":
        B[3, 7] = np.nan
        nb[7] = np.nan
    elif case == "inf norm":
        nb[::2] = np.inf
    elif case == "minus inf norm":
        nb[9] = -np.inf
    elif case == "zero norms":
        nb[:] = 0
    elif case == "huge center":
        B[:, 11] *= dtype(2.0 ** 70)
        nb = (B.astype(np.float64) ** 2).sum(0).astype(dtype)  # overflows to inf in FP32
    elif case == "inf row":
        A[17, 5] = np.inf
    elif case == "nan row":
        A[17, 5] = np.nan
    else:
        B[:] = B[:, :1]
        nb[:] = nb[0]
    with np.errstate(all="ignore"):
        want = exact_labels(A, B, nb)
    got = closest(km, torch_cuda, A, B, nb)
    keep = np.ones(n, bool)
    if case == "inf row":
        keep[17] = False  # infinite values: the entry's label is a tie among infinities
    assert np.array_equal(got[keep], want[keep])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("m,d,k,scale", [(1, 1, 1, 1.0), (70_001, 128, 40, 1.0), (5_000, 30, 7, 1.0),
                                         (3_000, 12, 5, 1e-18), (3_000, 16, 5, 1e19), (999, 200, 3, 0.0),
                                         (2_000, 77, 2, 1e4)])
def test_compactness_and_norms(km, torch_cuda, dtype, m, d, k, scale):
    torch = torch_cuda
    rng = np.random.default_rng(m + d)
    X = (rng.standard_normal((m, d)) * scale).astype(dtype)
    C = (rng.standard_normal((k, d)) * scale).astype(dtype)
    lab = rng.integers(0, k, m).astype(np.int32)
    F = dtype == np.float32
    x, c, l = (torch.from_numpy(v).cuda() for v in (X, C, lab))
    out = torch.zeros(4, dtype=x.dtype, device="cuda")
    fn = km.CompactnessF if F else km.CompactnessD
    assert fn(0, m, True, d, k, x, l, c, out) == 0
    with np.errstate(over="ignore"):
        want = dtype(((X.astype(np.float64) - C.astype(np.float64)[lab]) ** 2).sum())
        rows = (X.astype(np.float64) ** 2).sum(1)
        cols = (X.astype(np.float64) ** 2).sum(0)
        # FP32 outputs are one rounding of (nearly) FP64 values; subnormal results keep absolute steps
        tol = dict(rtol=1.3e-7, atol=3e-45) if F else dict(rtol=1e-12, atol=0)
        np.testing.assert_allclose(out.cpu().numpy()[0], want, **tol)
        r = torch.zeros(m + 2, dtype=x.dtype, device="cuda")
        q = torch.zeros(d, dtype=x.dtype, device="cuda")
        assert (km.rowNormalizeF if F else km.rowNormalizeD)(2, m, d, x, r) == 0
        assert (km.colNormalizeF if F else km.colNormalizeD)(m, d, x, q) == 0
        np.testing.assert_allclose(r.cpu().numpy()[2:], rows.astype(dtype), **tol)
        np.testing.assert_allclose(q.cpu().numpy(), cols.astype(dtype), **tol)


@pytest.mark.parametrize("n,d,k", [(300, 8, 40), (33, 33, 70), (20_000, 64, 256), (200, 700, 9)])
@pytest.mark.parametrize("sign", [-1, 1])
def test_closest_centers_beyond_fp32_range(km, torch_cuda, n, d, k, sign):
    """Products that overflow FP32 with centers whose norms do not: every center's FP32 value is
    infinite, the FP64 values decide."""
    rng = np.random.default_rng(n + k)
    A = (1e20 * rng.uniform(0.5, 2.0, (n, d))).astype(np.float32)
    B = (sign * min(1.0, (64 / d) ** 0.5) * rng.uniform(1e18, 2e18, (d, k))).astype(np.float32)
    nb = (B.astype(np.float64) ** 2).sum(0).astype(np.float32)
    assert np.isfinite(nb).all()
    assert np.array_equal(closest(km, torch_cuda, A, B, nb), exact_labels(A, B, nb))


# Rows whose squared norm lies within 2^-46 of the middle between two FP32 numbers.
NEARLY_MIDWAY = [
    "0x1.bd8ff8p-4 0x1.ba67f4p-1 -0x1.b7f980p-4 -0x1.888288p-2 0x1.6cec4cp-10 0x1.2c0592p-1 0x1.b69d1ap-3 0x1.ad9c86p-1",
    "-0x1.3c572ap-1 0x1.5c5984p-1 0x1.578ce2p-5 0x1.e65b9cp-3 -0x1.3e26a4p-3 0x1.7a3870p-1 0x1.f23a48p-2 0x1.2ecfd0p-1",
    "0x1.96e9a4p-1 -0x1.2a8184p-1 -0x1.c481b8p-1 0x1.743e32p-3 0x1.ba0478p-4 0x1.670c88p-2 0x1.6dc126p-2 0x1.e6b306p-1",
    "0x1.b85822p-1 -0x1.fa089ap-1 -0x1.099144p-3 -0x1.6c51ecp-1 0x1.c4a526p-1 0x1.ede244p-3 0x1.1f59cap-2 0x1.0ccc0ep+0",
    "0x1.2d6fdap-1 -0x1.8dcd54p-1 -0x1.c2f75ap-2 -0x1.428910p-1 -0x1.8a8634p-1 -0x1.055c46p-2 0x1.567434p-2 0x1.7f29aap-1",
    "-0x1.6c7afcp-1 0x1.00789ap-4 0x1.2265c2p-1 -0x1.c585fcp-1 0x1.1db252p-4 -0x1.abedd8p-1 0x1.e670f6p-2 0x1.3eff7cp-1",
]


def test_row_norms_are_the_fp64_sums_rounded(km, torch_cuda):
    from fractions import Fraction
    rows = np.array([[float.fromhex(v) for v in r.split()] for r in NEARLY_MIDWAY], np.float32)
    want = []
    for r in rows:
        s = sum(Fraction(float(v)) ** 2 for v in r)
        near = np.float32(float(s))
        want.append(min((near, np.nextafter(near, np.float32(0)), np.nextafter(near, np.float32(9))),
                        key=lambda c: abs(Fraction(float(c)) - s)))
    X = np.tile(rows, (50, 1))  # whole warps of them, and beside ordinary rows
    X[7::11] = np.random.default_rng(1).standard_normal(X[7::11].shape)
    out = torch_cuda.zeros(len(X), device="cuda")
    assert km.rowNormalizeF(0, len(X), 8, torch_cuda.from_numpy(X).cuda(), out) == 0
    got = out.cpu().numpy()
    for i, w in enumerate(np.tile(np.array(want, np.float32), 50)):
        if i % 11 != 7:
            assert got[i] == w, i


@pytest.mark.parametrize("n", [8192, 1000, 8190])  # 16 bytes a lane, and one element a lane
@pytest.mark.parametrize("big,small", [(4096.0, 0.9), (4096.0, 0.47), (1000.0, 0.1)])
def test_compactness_of_wide_rows(km, torch_cuda, n, big, small):
    """The running FP64 sum (the value behind out[0]) of rows whose squares all round the same way below
    one large square: within the 2^-35 of a lane's 128 terms, however wide the rows."""
    torch = torch_cuda
    X = np.full((64, n), small, np.float32)
    X[::32, :128] = big
    out = torch.zeros(6, device="cuda")
    lab = torch.zeros(64, dtype=torch.int32, device="cuda")
    c = torch.zeros((1, n), device="cuda")
    assert km.CompactnessF(0, 64, True, n, 1, torch.from_numpy(X).cuda(), lab, c, out) == 0
    acc = float(out.cpu().numpy()[2:4].copy().view(np.float64)[0])
    x = X.astype(np.float64)
    want = float(np.sum(np.sort((x * x).ravel())))
    assert abs(acc - want) <= 2.0 ** -35 * want


@pytest.mark.parametrize("n", [129, 2047, 4095, 4097, 8193])  # around 32 lanes of 128 terms, unaligned rows
@pytest.mark.parametrize("m", [1, 70])
def test_compactness_of_unaligned_wide_rows(km, torch_cuda, n, m):
    """The running FP64 sum where a row ends within, at and past the terms a lane adds up before it
    widens them: within the 2^-35 of these terms."""
    torch = torch_cuda
    rng = np.random.default_rng(n)
    X = rng.uniform(0.5, 900.0, (m, n)).astype(np.float32)
    C = rng.uniform(0.5, 900.0, (3, n)).astype(np.float32)
    lab = rng.integers(0, 3, m).astype(np.int32)
    out = torch.zeros(6, device="cuda")
    x, c, l = (torch.from_numpy(v).cuda() for v in (X, C, lab))
    assert km.CompactnessF(0, m, True, n, 3, x, l, c, out) == 0
    acc = float(out.cpu().numpy()[2:4].copy().view(np.float64)[0])
    want = float(((X.astype(np.float64) - C.astype(np.float64)[lab]) ** 2).sum())
    assert abs(acc - want) <= 2.0 ** -35 * want


def spoiled_rows(rng, n, d, k):
    """Rows with one element near FP32's largest number: every bound is infinite and every tensor-core
    key infinite or NaN; a key that stays infinite is one of a multiple of 32."""
    C = rng.uniform(-1000, 1000, (k, d)).astype(np.float32)
    X = C[rng.integers(0, k, n)] + rng.standard_normal((n, d)).astype(np.float32)
    rows = rng.choice(n, 60, replace=False)
    X[rows, rng.integers(0, d, 60)] = rng.choice([3e38, -3e38, 1e38], 60)
    return X, C, rows


@pytest.mark.parametrize("n,d,k", [(20_000, 64, 256), (30_000, 161, 115), (300, 40, 70)])
def test_closest_centers_of_rows_near_the_largest_number(km, torch_cuda, n, d, k):
    X, C, _ = spoiled_rows(np.random.default_rng(n), n, d, k)
    B = np.ascontiguousarray(C.T)
    nb = (B.astype(np.float64) ** 2).sum(0).astype(np.float32)
    assert np.array_equal(closest(km, torch_cuda, X, B, nb), exact_labels(X, B, nb))


@pytest.mark.parametrize("tier", ["BF16X3", "BF16", "FP32"])
@pytest.mark.parametrize("n,d,k", [(20_000, 64, 256), (70_000, 100, 115)])
def test_lloyd_with_rows_near_the_largest_number(km, orc, torch_cuda, tier, n, d, k):
    X, C, rows = spoiled_rows(np.random.default_rng(n), n, d, k)
    for flip in (1, -1):  # the sign decides which centers' keys are +inf
        Y = X * np.float32(flip)
        want = orc.lloyd(Y, C, 1, empty_policy=1)
        got = km.lloyd(Y, k, init=C, max_iters=1, assign_tier=getattr(km, "ASSIGN_" + tier), empty_policy=1)
        assert np.array_equal(got.labels, want[2])


@pytest.mark.parametrize("m", [1, 2, 3, 9, 16, 17, 40, 128, 700])
def test_column_norms_no_further_off_than_one_chain(km, torch_cuda, m):
    """colNormalizeD against exact sums: up to 16 rows the FP64 FMA chain over the rows itself, beyond
    no larger an error (root mean square over the columns) than that chain's."""
    from fractions import Fraction
    n = 600
    X = np.random.default_rng(m).standard_normal((m, n))
    out = torch_cuda.zeros(n, dtype=torch_cuda.float64, device="cuda")
    assert km.colNormalizeD(m, n, torch_cuda.from_numpy(X).cuda(), out) == 0
    got = out.cpu().numpy()
    chain, exact = np.empty(n), []
    for j in range(n):
        c, e = 0.0, Fraction(0)
        for v in X[:, j]:
            q = Fraction(float(v)) ** 2
            c = float(q + Fraction(c))
            e += q
        chain[j] = c
        exact.append(e)
    if m <= 16:
        assert np.array_equal(got, chain)
    else:
        def rms(v):
            return np.sqrt(np.mean([float((Fraction(float(a)) - e) / e) ** 2 for a, e in zip(v, exact)]))
        assert rms(got) <= rms(chain)
