"""fg_dense_gemm_nt where its tiles and its operand swap can go wrong: row- and column-major C
(the row-major product is computed as its transpose), ragged tiles of 128 x 64, K at the edges of
the exact chunk (170) and of its pieces (160), the triangular update, alpha and beta.

The bound is the header's: |error| <= k 2^-53 max_l|A_il| max_l|B_jl| plus the roundings of the
update, against an FP64 product accumulated in extended precision on the CPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fempar_gb300 as fg
    from fempar_gb300 import build, dense
    build.build()
    return fg.Context(0), dense, torch


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (127, 65, 16), (128, 64, 17), (129, 63, 160), (300, 130, 170),
                                   (130, 300, 171), (64, 400, 321), (378, 1000, 162)])
@pytest.mark.parametrize("layout", ["row", "col", "strided"])
def test_product(env, m, n, k, layout):
    ctx, dense, torch = env
    rng = np.random.default_rng(m * 1000 + n + k)
    A = rng.standard_normal((m, k)) * np.exp(rng.uniform(-6, 6, size=(m, 1)))
    B = rng.standard_normal((n, k)) * np.exp(rng.uniform(-6, 6, size=(n, 1)))
    C0 = rng.standard_normal((m, n))
    ref = (A.astype(np.longdouble) @ B.astype(np.longdouble).T)
    scale = np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()

    def out():
        if layout == "row":
            return torch.from_numpy(C0.copy()).cuda()
        if layout == "col":
            return torch.from_numpy(np.ascontiguousarray(C0.T)).cuda().t()
        big = torch.zeros((2 * m, 3 * n), dtype=torch.float64, device="cuda")
        v = big[::2, ::3]
        v.copy_(torch.from_numpy(C0))
        return v

    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (0.75, -2.0)):
        C = out()
        dense.gemm_nt(ctx, dA, dB, C, alpha=alpha, beta=beta)
        want = alpha * ref + beta * C0
        # the product's bound, and two FP64 roundings of the update
        tol = abs(alpha) * k * 2.0 ** -53 * scale + 2.0 ** -52 * (np.abs(alpha * ref) + np.abs(beta * C0))
        assert np.all(np.abs(C.cpu().numpy() - want) <= tol), (alpha, beta)


@pytest.mark.parametrize("m,k", [(64, 16), (129, 128), (260, 170), (200, 200)])
def test_lower(env, m, k):
    ctx, dense, torch = env
    rng = np.random.default_rng(m + k)
    A = rng.standard_normal((m, k))
    C0 = rng.standard_normal((m, m))
    for col in (False, True):
        C = torch.from_numpy(np.ascontiguousarray(C0.T if col else C0)).cuda()
        C = C.t() if col else C
        dense.gemm_nt(ctx, torch.from_numpy(A).cuda(), None, C, alpha=-1.0, beta=1.0, lower=True)
        got = C.cpu().numpy()
        ref = A.astype(np.longdouble) @ A.astype(np.longdouble).T
        want = C0 - ref
        scale = np.abs(A).max(1)[:, None] * np.abs(A).max(1)[None, :]
        tol = k * 2.0 ** -53 * scale + 2.0 ** -52 * (np.abs(ref) + np.abs(C0))
        low = np.tril(np.ones((m, m), dtype=bool))
        assert np.all(np.abs(got - want)[low] <= tol[low])
        assert np.array_equal(got[~low], C0[~low])


@pytest.mark.parametrize("p,q", [(0, 0), (-700, -350), (520, 503), (40, -31)])
def test_sum_to_fp64(env, p, q):
    """The integer sum's way to FP64, exactly: sums that cancel down to the last digit, of both
    signs, zero, and results that are subnormal or close to overflow (rows are cut 56 bits below a
    power of two above their largest value, so 2^-i for i <= 53 beside 1 is exact)."""
    ctx, dense, torch = env
    i = np.arange(54)
    A = np.zeros((109, 3))
    A[:54], A[54:108] = [1.0, -1.0, 0.0], [1.0, -1.0, 0.0]
    A[:54, 2], A[54:108, 2] = np.ldexp(1.0, -i), -np.ldexp(1.0, -i)
    B = np.ones((65, 3))
    for sign in (1.0, -1.0):
        C = dense.gemm_nt(ctx, torch.from_numpy(np.ldexp(A, p)).cuda(), torch.from_numpy(np.ldexp(B, q)).cuda(),
                          torch.zeros((109, 65), dtype=torch.float64, device="cuda"), alpha=sign)
        want = sign * np.ldexp(A[:, 2], p + q)
        assert np.array_equal(C.cpu().numpy(), np.repeat(want[:, None], 65, axis=1))


@pytest.mark.parametrize("m,n,k", [(300, 64, 64), (300, 130, 33), (129, 65, 128), (64, 200, 20), (700, 700, 64)])
def test_lower_rectangular(env, m, n, k):
    """The tiles of a triangular update of another shape than square: fewer columns than rows (a panel's),
    more, and the ragged last row and column of tiles; elements above the diagonal stay as they are."""
    ctx, dense, torch = env
    rng = np.random.default_rng(m + n + k)
    A, B, C0 = rng.standard_normal((m, k)), rng.standard_normal((n, k)), rng.standard_normal((m, n))
    C = torch.from_numpy(np.ascontiguousarray(C0.T)).cuda().t()
    dense.gemm_nt(ctx, torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), C, alpha=-1.0, beta=1.0, lower=True)
    got = C.cpu().numpy()
    ref = A.astype(np.longdouble) @ B.astype(np.longdouble).T
    scale = np.abs(A).max(1)[:, None] * np.abs(B).max(1)[None, :]
    tol = k * 2.0 ** -53 * scale + 2.0 ** -52 * (np.abs(ref) + np.abs(C0))
    lower = np.tril(np.ones((m, n), dtype=bool))
    assert np.all(np.abs(got - (C0 - ref))[lower] <= tol[lower])
    assert np.array_equal(got[~lower], C0[~lower])
