"""The factorisation inside a 128-column panel (BDDC set-up) keeps FP64's accuracy for entries far below
their row's largest: one subdomain of at most 128 dofs, whose FP64 apply is A^-1 r by one panel.

Graded coefficients (10^-x per cell of x) and unit loads: componentwise errors of the solutions against
80-bit elimination, the largest of three loads per matrix.  Bar: eight times LAPACK's own FP64 Cholesky solve
of the same matrix, at least 8 n 2^-53 (an update by seven 8-bit digits cut at 2^-54 of a row's largest
entry is off by up to 20 times LAPACK's there; eight digits are within two)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fg():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fempar_gb300 as fg
    from fempar_gb300 import build
    build.build()
    return fg


def exact_solve(A, r):
    """Cholesky and two substitutions in the host's long double (80 bits on x86, 128 on Arm)."""
    A, y = A.astype(np.longdouble), r.astype(np.longdouble)
    n = len(A)
    L = np.zeros_like(A)
    for k in range(n):
        L[k, k] = np.sqrt(A[k, k])
        L[k + 1:, k] = A[k + 1:, k] / L[k, k]
        A[k + 1:, k + 1:] -= np.outer(L[k + 1:, k], L[k + 1:, k])
    for k in range(n):
        y[k] /= L[k, k]
        y[k + 1:] -= L[k + 1:, k] * y[k]
    for k in range(n - 1, -1, -1):
        y[k] = (y[k] - L[k + 1:, k] @ y[k + 1:]) / L[k, k]
    return y


@pytest.mark.parametrize("n,order,grade", [((7, 3, 3), 1, 1.0), ((7, 3, 3), 1, 0.5), ((6, 3, 4), 1, 1.5), ((3, 2, 1), 2, 2.0)])
def test_one_panel(fg, n, order, grade):
    import scipy.linalg
    import scipy.sparse as sp
    import torch
    ctx = fg.Context(0)
    coef = np.array([10.0 ** (-grade * (c % n[0])) for c in range(int(np.prod(n)))])
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=order, dirichlet_ids=[1, 3, 5, 7, 13, 15, 17, 19, 25])
    N = space.num_free_dofs
    assert N <= 128
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(cell_coef=coef, source_fn=fg.FG_FN_CONST, fn_param=[1.0])).compute()
    irp, ja, val = op.get_matrix(symmetric_storage=False, one_based=False)
    A = sp.csr_matrix((val, ja, irp), shape=(N, N)).toarray()
    M = fg.MLBDDC(op, nsub=(1, 1, 1))
    chol = scipy.linalg.cho_factor(A, lower=True)
    mine = lapack = 0.0
    for where in (0, N // 2, N - 1):
        r = np.zeros(N)
        r[where] = 1.0
        t = exact_solve(A, r)
        d = torch.from_numpy(r).cuda()
        z = torch.empty_like(d)
        torch.cuda.synchronize()
        M.apply_device(d, z, fg.FG_FP64)
        torch.cuda.synchronize()
        err = lambda x: float((np.abs(x - t) / np.abs(t)).max())
        mine, lapack = max(mine, err(z.cpu().numpy())), max(lapack, err(scipy.linalg.cho_solve(chol, r)))
    assert mine <= 8 * max(lapack, N * 2.0 ** -53), (mine, lapack)
    M.close()
