"""The rare paths and edges of the register-row, tensor-core, triangular-solve and
emulated-format kernels: pivots that need the exact comparison, divisions outside the
shared-reciprocal range, zero pivots over columns that are not plain zeros, ragged
orders, partial passes of right-hand sides, binary16 storage."""
import numpy as np
import pytest

from conftest import load_pkg

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

tsdx = load_pkg()
capi = load_pkg("capi")
device = load_pkg("device")
M = load_pkg("matrices")


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def same(a, b):
    """Bit-identical, NaN where the other has NaN."""
    iv = {2: np.uint16, 4: np.uint32, 8: np.uint64}[a.dtype.itemsize]
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return bool(((a.view(iv) == b.view(iv)) | (np.isnan(a) & np.isnan(b))).all())


def odd_matrices(n, dtype, seed):
    r = np.random.default_rng(seed)
    f32 = dtype == np.float32
    A = r.standard_normal((14, n, n)).astype(dtype)
    c = n // 2
    A[0] *= dtype(1e-30 if f32 else 1e-200)                     # pivots below the range
    A[1] *= dtype(1e33 if f32 else 1e200)                       # and above it
    A[2, ::2] *= dtype(1e-25 if f32 else 1e-190)                # tiny multipliers
    A[3, :, c] = -0.0                                           # a zero pivot over -0
    A[4, :, c] = 0.0
    A[4, -1, c] = np.nan                                        # and over a NaN
    A[5, 0, 0] = np.nan
    A[6, -1, 0] = np.inf
    A[7] = r.integers(-1, 2, (n, n))                            # ties and zeros
    A[8] = np.eye(n)[r.permutation(n)]
    A[9, 0, 0] = np.nextafter(dtype(4), dtype(0))               # an all-ones significand
    A[10, 0, 0] = -np.nextafter(dtype(4), dtype(0))
    A[11] = np.where(r.random((n, n)) < 0.6, 0.0, A[11])
    A[12] = 0.0
    for i in (9, 10):
        A[i, 1:, 0] = (r.integers(1, 16, n - 1) / 8.0).astype(dtype)
    return A


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [2, 4, 7, 8, 16, 21, 24, 29, 32, 40, 45, 48, 61, 64])
def test_odd_pivots_bit_exact(oracle, n, dtype):
    A = odd_matrices(n, dtype, 900 + n)
    LU, piv, info = (t.cpu().numpy() for t in (lambda a: (a, *device.getrf(a)))(dev(A)))
    LUo, pivo, infoo = oracle.lu(A, "scalar")
    assert np.array_equal(info, infoo) and np.array_equal(piv, pivo)
    for i in range(len(A)):
        assert same(LU[i], LUo[i]), i


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [2, 4, 7, 8, 16, 21, 24, 29, 32, 40, 45, 48, 61, 64])
@pytest.mark.parametrize("nrhs", [1, 3, 8])
def test_odd_pivots_with_right_hand_sides(oracle, n, nrhs, dtype):
    """The same pivots under gesv, in warps shared with healthy matrices: factors, pivots and
    info as the oracle's, and the healthy ones' solutions as in a batch of their own."""
    odd = odd_matrices(n, dtype, 300 + n)
    r = np.random.default_rng(n * 5 + nrhs)
    good = M.general(r, len(odd), n, 1e2).astype(dtype)
    A = np.empty((2 * len(odd), n, n), dtype)
    A[0::2], A[1::2] = odd, good
    B = r.standard_normal((len(A), n, nrhs)).astype(dtype)
    a, b = dev(A), dev(B)
    piv, info = (t.cpu().numpy() for t in device.gesv(a, b))
    LUo, pivo, infoo = oracle.lu(A, "scalar")
    assert np.array_equal(info, infoo) and np.array_equal(piv, pivo) and same(a.cpu().numpy(), LUo)
    a, x = dev(good), dev(B[1::2])
    device.gesv(a, x)
    assert same(b[1::2].cpu().numpy(), x.cpu().numpy())
    X, B64 = x.cpu().numpy().astype(np.float64), B[1::2].astype(np.float64)
    num = np.linalg.norm(B64 - good.astype(np.float64) @ X, axis=1)
    den = np.linalg.norm(good.astype(np.float64), axis=(1, 2))[:, None] * np.linalg.norm(X, axis=1) + np.linalg.norm(B64, axis=1)
    assert (num / den).max() <= 8 * n * np.finfo(dtype).eps / 2


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("sched", [0, 15])
def test_odd_pivots_in_a_stream(oracle, sched, dtype):
    """Every order, odd and healthy matrices and both kinds in the same units: factors, pivots
    and info as the oracle's, the healthy ones' solutions as in the dense batch."""
    st = load_pkg("stream")
    r = np.random.default_rng(77 + sched)
    count = 64 * 24
    n = np.tile(np.arange(1, 65, dtype=np.int32), 24)
    nrhs = r.choice([0, 1, 3, 8], count).astype(np.int32)
    kind = r.integers(0, 2, count).astype(np.int8)
    order = r.permutation(count)
    n = n[order]
    mats, healthy = [], []
    for i in range(count):
        m, ok = int(n[i]), not kind[i] or i % 3 == 0
        if not kind[i]:
            mats.append(M.spd(r, 1, m, 1e2)[0].astype(dtype))
        elif ok or m < 2:
            mats.append(M.general(r, 1, m, 1e2)[0].astype(dtype))
        else:
            mats.append(odd_matrices(m, dtype, int(i))[int(r.integers(14))])
        healthy.append(ok or m < 2)
    rhs = [r.standard_normal((int(m), int(k))).astype(dtype) for m, k in zip(n, nrhs)]
    plan = st.StreamPlan(n, nrhs, kind, dtype=torch.float32 if dtype == np.float32 else torch.float64)
    plan.sched = sched
    plan.load(dev(np.concatenate([a.ravel() for a in mats])), dev(np.concatenate([b.ravel() for b in rhs])))
    plan.launch()
    A, B, piv, info = (t.cpu().numpy() for t in (plan.A, plan.B, plan.piv, plan.info))
    aoff, boff, poff = (t.cpu().numpy() for t in (plan.aoff, plan.boff, plan.poff))
    for i in range(count):
        m, k = int(n[i]), int(nrhs[i])
        F = A[aoff[i]:aoff[i] + m * m].reshape(1, m, m)
        if kind[i]:
            Fo, po, io = oracle.lu(mats[i][None], "scalar")
            assert np.array_equal(piv[poff[i]:poff[i] + m], po[0]), i
        else:
            Fo, io = oracle.cholesky(mats[i][None], "simd")
        assert info[i] == io[0] and same(F, Fo), i
        if healthy[i] and k:
            a, b = dev(mats[i][None]), dev(rhs[i][None])
            device.gesv(a, b) if kind[i] else device.posv(a, b)
            X, Y = B[boff[i]:boff[i] + m * k].reshape(m, k), b[0].cpu().numpy()
            assert same(X, Y), i


def step_check(a, b):
    out = [torch.empty_like(a) for _ in range(4)]
    capi.check(capi.call("tsdx_internal_step_check_" + ("f32" if a.dtype == torch.float32 else "f64"), capi.ptr(a), capi.ptr(b),
                         *map(capi.ptr, out), a.numel(), capi.stream_ptr()))
    q, q_ieee, y, y_ieee = (t.view(torch.int32 if a.dtype == torch.float32 else torch.int64) for t in out)
    assert torch.equal(y, y_ieee) and torch.equal(q, q_ieee)


@pytest.mark.parametrize("exponent", [-100, -99, -50, -1, 0, 1, 64, 99, 100])
def test_step_division_float32(exponent):
    """Every significand as the divisor, numerators from its size down to the smallest."""
    g = torch.Generator(device="cuda").manual_seed(exponent + 200)
    sig = torch.arange(1 << 23, device="cuda", dtype=torch.int32)
    for sign in (0, -(1 << 31)):
        b = (sig | ((127 + exponent) << 23) | sign).view(torch.float32)
        for low in (0, 30, 130):
            u = torch.rand(1 << 23, device="cuda", generator=g) * 2 - 1
            a = (b * u) * torch.exp2(-torch.randint(0, low + 1, (1 << 23,), device="cuda", generator=g).float())
            a[::1001] = 0.0
            a[1::1001] = -0.0
            a[2::1001] = b[2::1001]
            step_check(a, b)


@pytest.mark.parametrize("exponent", [-900, -899, -600, -1, 0, 1, 400, 899, 900])
def test_step_division_float64(exponent):
    """Random significands and those next to all ones and to one, numerators likewise."""
    n = 1 << 24
    g = torch.Generator(device="cuda").manual_seed(exponent + 2000)
    ones = (1 << 52) - 1
    for rep in range(4):
        sig = torch.randint(0, ones + 1, (n,), device="cuda", generator=g, dtype=torch.int64)
        near = torch.randint(0, 64, (n // 4,), device="cuda", generator=g, dtype=torch.int64)
        sig[: n // 4] = ones - near * (rep % 2)
        sig[n // 4: n // 2] = near
        b = (sig | ((1023 + exponent) << 52)).view(torch.float64) * (1 - 2 * (rep // 2))
        a = b * (torch.rand(n, device="cuda", generator=g, dtype=torch.float64) * 2 - 1)
        a *= torch.exp2(-torch.randint(0, (1, 60, 950, 1000)[rep] + 1, (n,), device="cuda", generator=g).double())
        a[::1001] = 0.0
        a[1::1001] = -0.0
        a[2::1001] = b[2::1001]
        step_check(a, b)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [3, 4, 8, 16, 24, 31, 32, 40, 45, 48, 56, 61, 64])
def test_scaled_matrices_bit_exact(oracle, n, dtype):
    """Powers of two put pivots and numerators on either side of the range of the shared
    reciprocal division: whole matrices, single rows and columns, and D S D of an SPD
    matrix; with -0 among the numerators, ties, and symmetric matrices that are not
    dominated by their diagonal."""
    r = np.random.default_rng(600 + n)
    edges = (99, 100, 101, 119, 121) if dtype == np.float32 else (899, 900, 901, 600, 400, 500)
    A, S = [], []
    for e in edges:
        for sign in (1, -1):
            X = r.standard_normal((n, n))
            Q = X @ X.T / n + 0.2 * np.eye(n)
            Z = np.where(r.random((n, n)) < 0.3, -0.0, X)
            d, col = np.ones(n), np.ones(n)
            d[r.integers(n)] = col[r.integers(n)] = 2.0 ** (sign * e)
            half = 2.0 ** r.integers(-(e // 2), e // 2 + 1, n)
            A += [X * 2.0 ** (sign * e), X * d[:, None], X * col, Z, np.rint(2 * X) * 2.0 ** (sign * (e // 2))]
            S += [Q * 2.0 ** (sign * e), Q * half[:, None] * half, np.where(np.abs(Q) < 0.3, -0.0, Q) + np.diag(np.full(n, n + 0.0)),
                  X + X.T, Q * np.sqrt(d)[:, None] * np.sqrt(d)]
    with np.errstate(over="ignore", under="ignore"):
        A, S = np.stack(A).astype(dtype), np.stack(S).astype(dtype)
    a = dev(A)
    piv, info = device.getrf(a)
    LUo, pivo, infoo = oracle.lu(A, "scalar")
    assert np.array_equal(info.cpu().numpy(), infoo) and np.array_equal(piv.cpu().numpy(), pivo)
    assert same(a.cpu().numpy(), LUo)
    s = dev(S)
    info = device.potrf(s).cpu().numpy()
    Lo, infoo = oracle.cholesky(S, "simd")
    assert np.array_equal(info, infoo)
    ok = infoo == 0
    assert ok.any() and same(s.cpu().numpy()[ok], Lo[ok])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 47, 49, 64])
@pytest.mark.parametrize("nrhs", [2, 4, 5, 8, 16, 17])
def test_solves_from_factor(oracle, n, nrhs, dtype):
    r = np.random.default_rng(n * 31 + nrhs)
    A = M.general(r, 9, n, 1e2).astype(dtype)
    S = M.spd(r, 9, n, 1e2).astype(dtype)
    B = r.standard_normal((9, n, nrhs)).astype(dtype)
    LU, piv, _ = oracle.lu(A, "scalar")
    L, _ = oracle.cholesky(S, "simd")
    bad = piv.astype(np.int32).copy()
    bad[0, -1] = n            # a pivot that names no row is ignored: the last swap is a no-op anyway
    bad[1, -1] = -1
    for mats, run in ((A, lambda b: device.getrs(dev(LU), dev(bad), b)), (S, lambda b: device.potrs(dev(L), b))):
        b = dev(B)
        run(b)
        X, M64, B64 = b.cpu().numpy().astype(np.float64), mats.astype(np.float64), B.astype(np.float64)
        num = np.linalg.norm(B64 - M64 @ X, axis=1)
        den = np.linalg.norm(M64, axis=(1, 2))[:, None] * np.linalg.norm(X, axis=1) + np.linalg.norm(B64, axis=1)
        assert (num / den).max() <= 8 * n * np.finfo(dtype).eps / 2


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [1, 2, 8, 15, 16, 17, 24, 31, 47, 63, 64])
@pytest.mark.parametrize("nrhs", [1, 3, 8, 11, 17])
def test_solves_with_non_finite_right_hand_sides(oracle, n, nrhs, dtype):
    """Infinities, NaN and (potrs) a zero on the diagonal of L leave the same pattern of
    finite, infinite and NaN entries as the oracle's solve, whose terms are the same; the
    other columns keep the bits that they have without them."""
    r = np.random.default_rng(n * 37 + nrhs)
    A = M.general(r, 8, n, 1e2).astype(dtype)
    LU, piv, _ = oracle.lu(A, "scalar")
    L, _ = oracle.cholesky(M.spd(r, 8, n, 1e2).astype(dtype), "simd")
    B = r.standard_normal((8, n, nrhs)).astype(dtype)
    bad = B.copy()
    for i in range(8):
        bad[i, r.integers(n), i % nrhs] = (np.inf, -np.inf, np.nan)[i % 3]
    zero = L.copy()
    zero[3:, n // 2, n // 2] = 0.0
    for F, G, solve in ((LU, LU, lambda f, b: device.getrs(dev(f), dev(piv), b)), (L, zero, lambda f, b: device.potrs(dev(f), b))):
        good, x = dev(B), dev(bad)
        solve(F, good)
        solve(G, x)
        X, clean = x.cpu().numpy(), good.cpu().numpy()
        with np.errstate(all="ignore"):
            want = oracle.lu_solve(LU, piv, bad) if F is LU else oracle.cholesky_solve(zero, bad)
        assert np.array_equal(np.isnan(X), np.isnan(want))
        assert np.array_equal(X[np.isinf(X)], want[np.isinf(want)])
        for i in range(3 if F is L else 8):
            keep = [c for c in range(nrhs) if c != i % nrhs]
            assert same(X[i][:, keep], clean[i][:, keep])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,batch", [(1, 120_001), (2, 120_001), (3, 120_001), (4, 120_001), (5, 60_001), (7, 60_001), (8, 60_001),
                                     (9, 30_001), (11, 30_001), (12, 30_001), (13, 6_001), (16, 6_001), (17, 6_001), (24, 6_001), (33, 6_001), (40, 6_001),
                                     (56, 6_001), (63, 6_001)])
@pytest.mark.parametrize("nrhs", [1, 2, 5, 9])
def test_solves_of_large_batches(oracle, n, batch, nrhs, dtype):
    """More matrices than the resident warps hold, every warp of a block and every matrix of
    a warp: seven systems repeated over the batch, each copy with the bits of the first,
    and the first ones within the bound of test_solves_from_factor."""
    r = np.random.default_rng(n * 41 + nrhs)
    A, S = M.general(r, 7, n, 1e2).astype(dtype), M.spd(r, 7, n, 1e2).astype(dtype)
    B = r.standard_normal((7, n, nrhs)).astype(dtype)
    LU, piv, _ = oracle.lu(A, "scalar")
    L, _ = oracle.cholesky(S, "simd")
    at = torch.arange(batch, device="cuda") % 7
    for mats, run in ((A, lambda i, b: device.getrs(dev(LU)[i], dev(piv)[i], b)), (S, lambda i, b: device.potrs(dev(L)[i], b))):
        b = dev(B)[at]
        run(at, b)
        bits = b.view(torch.int32 if dtype == np.float32 else torch.int64)
        assert torch.equal(bits, bits[:7][at])
        X, M64, B64 = b[:7].cpu().numpy().astype(np.float64), mats.astype(np.float64), B.astype(np.float64)
        num = np.linalg.norm(B64 - M64 @ X, axis=1)
        den = np.linalg.norm(M64, axis=(1, 2))[:, None] * np.linalg.norm(X, axis=1) + np.linalg.norm(B64, axis=1)
        assert (num / den).max() <= 8 * n * np.finfo(dtype).eps / 2


@pytest.mark.parametrize("spd", [False, True])
@pytest.mark.parametrize("n", [5, 17, 40, 64])
def test_refinement_of_a_large_batch_of_mixed_tiers(n, spd):
    """Several rounds of full blocks whose warps take different tiers, float64 ones that leave
    the round at once among them: every copy of a system with its tier has the bits of the
    first."""
    r = np.random.default_rng(n + 7 * spd)
    batch = 7001
    A = (M.spd if spd else M.general)(r, 7, n, 1e3)
    b = r.standard_normal((7, n))
    at = torch.arange(batch, device="cuda")
    x = dev(b)[at % 7]
    tier = (at % 4).to(torch.int8)
    outs = (x, *device.ir(dev(A)[at % 7], x, spd, tier=tier))
    for t in outs:
        bits = t.view(torch.int64) if t.dtype == torch.float64 else t
        assert torch.equal(bits, bits[:28][at % 28])
    X = x[:28].cpu().numpy()
    num = np.linalg.norm(b[np.arange(28) % 7] - np.einsum("bij,bj->bi", A[np.arange(28) % 7], X), axis=1)
    den = np.linalg.norm(A, axis=(1, 2))[np.arange(28) % 7] * np.linalg.norm(X, axis=1) + np.linalg.norm(b, axis=1)[np.arange(28) % 7]
    assert (num / den).max() <= 8 * n * 2.0 ** -53


def test_metrics_from_several_threads():
    """Calls of different orders side by side, each thread on its own stream: every one
    succeeds (a kernel's shared-memory limit belongs to the function, so no call may lower
    it under another's launch) and gives what it gives alone."""
    import threading
    r = np.random.default_rng(4)
    work, errors = [], []
    for n in (64, 40, 64, 40):  # one kernel, 6 and 8 matrices a block
        A = dev(r.standard_normal((900, n, n)))
        F = A.clone()
        piv, _ = device.getrf(F)
        work.append((A, F, piv, device.lu_backward_error(A, F, piv)))
    torch.cuda.synchronize()
    start = threading.Barrier(len(work))

    def loop(A, F, piv, want):
        try:
            out, stream = torch.empty_like(want), torch.cuda.Stream()
            args = (capi.ptr(A), capi.ptr(F), capi.ptr(piv), A.shape[-1], A.shape[0], capi.ptr(out), capi.stream_ptr(stream))
            start.wait()
            for _ in range(4000):
                capi.check(capi.call("tsdx_cuda_lu_backward_error_f64", *args), "lu_backward_error")
            stream.synchronize()
            assert torch.equal(out, want)
        except Exception as e:
            errors.append(e)
    threads = [threading.Thread(target=loop, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("n", [20, 33, 64])
def test_metrics_keep_double_double_sums(n):
    """Sums whose remainder stands 105 bits below their largest term, after n - 8 roundings
    of the high part in one direction: exact in double-double, which renormalises at each
    term; lost in a low part that is a plain running sum."""
    from oracle import exact_metrics as X
    v = np.concatenate([[2.0 ** 53], np.full(n - 9, 0.75), np.full(5, 2.0 ** -52), [-2.0 ** 53, -0.75 * (n - 9)]])[:n]
    assert len(v) == n - 1
    A = np.zeros((1, n, n))
    A[0, -1, :-1] = v
    x, b = np.ones((1, n)), np.zeros((1, n))
    got = device.solve_backward_error(dev(A), dev(x), dev(b)).cpu().numpy()
    want = X.solve_backward_error(A, x, b)
    assert want[0] > 0
    np.testing.assert_allclose(got, want, rtol=1e-13, atol=0)
    LU = A.copy()
    LU[0, :-1, -1] = 1.0
    P = np.zeros((1, n, n))
    P[0, :-1, -1] = 1.0
    piv = np.arange(n, dtype=np.int32)[None]
    got = device.lu_backward_error(dev(P), dev(LU), dev(piv)).cpu().numpy()
    np.testing.assert_allclose(got, X.lu_backward_error(P, LU, piv), rtol=1e-13, atol=0)


@pytest.mark.parametrize("n", [2, 31, 32, 33, 47, 64])
def test_metrics_of_large_batches(oracle, n):
    """Every warp and team of a block, and several rounds: each copy has the bits of the first,
    and the first ones the values of exact arithmetic."""
    from oracle import exact_metrics as X
    batch = 5003
    r = np.random.default_rng(n)
    A, S, b = M.general(r, 5, n, 1e3), M.spd(r, 5, n, 1e3), r.standard_normal((5, n))
    LU, piv, _ = oracle.lu(A, "scalar")
    L, _ = oracle.cholesky(S, "simd")
    x = oracle.lu_solve(LU, piv, b[..., None])[..., 0]
    piv = piv.astype(np.int32)
    at = torch.arange(batch, device="cuda") % 5
    for got, want in ((device.lu_backward_error(dev(A)[at], dev(LU)[at], dev(piv)[at]), X.lu_backward_error(A[:2], LU[:2], piv[:2])),
                      (device.chol_backward_error(dev(S)[at], dev(L)[at]), X.chol_backward_error(S[:2], L[:2])),
                      (device.solve_backward_error(dev(A)[at], dev(x)[at], dev(b)[at]), X.solve_backward_error(A[:2], x[:2], b[:2]))):
        bits = got.view(torch.int64)
        assert torch.equal(bits, bits[:5][at])
        np.testing.assert_allclose(got[:2].cpu().numpy(), want, rtol=1e-12, atol=0)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64])
def test_binary16_storage_equals_cpu(n):
    r = np.random.default_rng(n)
    S = M.spd(r, 5, n, 10.0).astype(np.float16)
    G = r.standard_normal((5, n, n)).astype(np.float16)
    B = r.standard_normal((5, n, 3)).astype(np.float16)
    if n > 2:
        S[1, 1, 1] = -1.0
        G[1, :, 1] = 0.0
        G[2] = r.integers(-1, 2, (n, n))
    for f, X in ((tsdx.cholesky, S), (tsdx.lu, G)):
        got, want = f(X, backend="cuda"), f(X, backend="scalar")
        assert got[0].dtype == np.float16 and same(got[0], want[0])
        assert all(np.array_equal(a, b) for a, b in zip(got[1:], want[1:]))
    L, _ = tsdx.cholesky(S[2:], backend="scalar")
    assert same(tsdx.cholesky_solve(L, B[2:], backend="cuda"), tsdx.cholesky_solve(L, B[2:], backend="scalar"))
    LU, piv, _ = tsdx.lu(G[3:], backend="scalar")
    assert same(tsdx.lu_solve(LU, piv, B[3:], backend="cuda"), tsdx.lu_solve(LU, piv, B[3:], backend="scalar"))


@pytest.mark.parametrize("n", [1, 2, 4, 5, 8, 9])
@pytest.mark.parametrize("nrhs", [4, 5, 8, 11])
def test_posv_of_a_large_batch_equals_a_small_one(n, nrhs):
    """From 16,384 matrices on, float64 posv of orders 4 and 8 solves five or more right-hand
    sides from the factor: factors, info and solutions as the one-pass kernel's, failing
    pivots and non-finite entries included."""
    r = np.random.default_rng(n * 19 + nrhs)
    S = M.spd(r, 9, n, 1e3)
    S[1, n // 2, n // 2] = -1.0
    S[2] *= 1e200
    S[3, -1, 0] = np.nan
    S[4, 0, 0] = 0.0
    B = r.standard_normal((9, n, nrhs))
    B[5, 0, 0], B[6, -1, -1], B[7, 0] = np.inf, np.nan, -0.0
    want = (dev(S), dev(B))
    info = device.posv(*want)
    at = torch.arange(16384 + 5, device="cuda") % 9
    got = (dev(S)[at], dev(B)[at])
    big = device.posv(*got)
    assert torch.equal(big, info[at])
    for g, w in zip(got, want):
        assert same(g.cpu().numpy(), w[at].cpu().numpy())


@pytest.mark.parametrize("n", [3, 17, 33, 64])
@pytest.mark.parametrize("fmt", ["fp16", "bf16"])
def test_emulated_formats_of_large_batches(n, fmt):
    """More matrices than a wave of full blocks: five systems repeated, each copy with the bits
    of the CPU's result."""
    r = np.random.default_rng(n)
    batch = 12_001 if n < 40 else 6_001
    S = M.spd(r, 5, n, 10.0).astype(np.float32)
    G = r.standard_normal((5, n, n)).astype(np.float32)
    B = r.standard_normal((5, n, 2)).astype(np.float32)
    at = np.arange(batch) % 5
    for f, X in ((tsdx.cholesky, S), (tsdx.lu, G)):
        got, want = f(X[at], precision=fmt, backend="cuda"), f(X, precision=fmt, backend="scalar")
        assert same(got[0], want[0][at]) and all(np.array_equal(g, w[at]) for g, w in zip(got[1:], want[1:]))
    L, _ = tsdx.cholesky(S, precision=fmt, backend="scalar")
    LU, piv, _ = tsdx.lu(G, precision=fmt, backend="scalar")
    assert same(tsdx.cholesky_solve(L[at], B[at], precision=fmt, backend="cuda"),
                tsdx.cholesky_solve(L, B, precision=fmt, backend="scalar")[at])
    assert same(tsdx.lu_solve(LU[at], piv[at], B[at], precision=fmt, backend="cuda"),
                tsdx.lu_solve(LU, piv, B, precision=fmt, backend="scalar")[at])


def test_empty_batch_of_an_emulated_format_needs_no_pointers():
    for sfx in ("", "_f32", "_f16"):
        assert capi.call("tsdx_cuda_emu_factor_host" + sfx, 0, 1, None, 4, 0, None, None) == capi.TSDX_OK
        assert capi.call("tsdx_cuda_emu_solve_host" + sfx, 0, 1, None, None, 4, 0, None, 3) == capi.TSDX_OK
        assert capi.call("tsdx_cuda_emu_factor_host" + sfx, 0, 1, None, 4, 1, None, None) == capi.TSDX_ERR_NULL


def test_wide_host_solves_keep_little_device_memory():
    """400 MB of right-hand sides of small factors go through in chunks: what the calls leave
    allocated is bounded by the chunks, not by the right-hand sides."""
    n, batch, nrhs = 2, 32, 800_000
    F = np.broadcast_to(np.array([[2.0, 0.0], [1.0, 4.0]]), (batch, n, n)).copy()
    B = np.ones((batch, n, nrhs))
    B[:, 1] = np.arange(batch)[:, None]
    device.potrf(dev(np.eye(2)[None]))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    X = tsdx.cholesky_solve(F, B, precision="fp16", backend="cuda")
    assert free - torch.cuda.mem_get_info()[0] < 3 * (200 << 20)
    want = tsdx.cholesky_solve(F, B[..., :3].copy(), precision="fp16", backend="scalar")
    assert same(np.ascontiguousarray(X[..., [0, nrhs // 2, nrhs - 1]]), want)


@pytest.mark.parametrize("n", [1, 5, 32, 33, 64])
def test_features_of_zero_rows_have_no_negative_zero(n):
    sel = load_pkg("selector")
    r = np.random.default_rng(n)
    A = r.standard_normal((3, n, n))
    A[0] = 0.0
    A[1] = -0.0
    A[2, n // 2] = 0.0
    X = sel.features(dev(A), 1).cpu().numpy()
    assert not (np.signbit(X) & (X == 0.0)).any()


@pytest.mark.parametrize("batch", [1, 63, 64, 65, 600])
def test_training_gradient_of_partial_blocks(batch):
    """Against float64: float32 sums of at most 600 samples over 64 units carry a few
    hundred roundings of 2^-24 of the largest term; 2e-5 of the largest entry bounds them."""
    from oracle import selector_ref as R
    sel = load_pkg("selector")
    r = np.random.default_rng(batch)
    X = (r.standard_normal((batch, 24)) * 2 + 1).astype(np.float32)
    y = r.integers(0, 4, batch).astype(np.int8)
    s = sel.Selector(seed=3)
    grad, loss = s.loss_grad(dev(X), dev(y), torch.tensor([1.0, 2.0, 0.5, 0.7]))
    lo, g = R.loss_and_grad(s.params.cpu().numpy(), s.norm.cpu().numpy(), X, y, np.array([1.0, 2.0, 0.5, 0.7]))
    assert np.abs(grad.cpu().numpy() - g).max() <= 2e-5 * np.abs(g).max()
    assert abs(float(loss) - float(lo)) <= 2e-5 * abs(float(lo))
