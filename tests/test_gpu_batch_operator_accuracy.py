"""The batch solver's FP32 operator on smooth vectors, where products with the stiffness matrix cancel
to h^2 of their terms: with exact tables (small integers) the cancellation costs no accuracy of the step
length.  One iteration at order 1 from a smooth source gives x = alpha D^-1 b with
alpha = <b, D^-1 b> / <D^-1 b, A D^-1 b>, D^-1 b smooth.

Bound: x carries five FP32 roundings per node (b, its product with 1/D, 1/D, alpha and the update), 5 2^-24
= 3.0e-7 at the most, and the operator's error in alpha, under 2e-8 by emulation (4e-7 at 32 nodes in a
direction, and growing, with rounded entries)."""
import numpy as np
import pytest

from test_gpu_batch_apply import line_matrices

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fempar_gb300 as fg
    from fempar_gb300 import build
    build.build()
    return fg.Context(0), torch


@pytest.mark.parametrize("n", [33, 64, 128])
def test_step_length(env, n):
    ctx, torch = env
    from fempar_gb300.batch import BatchSolver
    F, q = n - 1, 2
    dev = torch.device("cuda", 0)
    xq = (np.arange(n)[:, None] + 0.5 * (1.0 + np.polynomial.legendre.leggauss(q)[0])).ravel() / n
    s = torch.from_numpy(np.sin(np.pi * xq)).to(dev)
    f = s[:, None, None] * s[:, None] * s                      # at the Gauss points, [z][y][x]
    flat = f.view(n, q, n, q, n, q).permute(0, 2, 4, 1, 3, 5).reshape(-1).contiguous()  # cell by cell
    x = torch.zeros(F ** 3, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    B = BatchSolver(ctx, [{"n": n, "order": 1, "coef": 1.3, "qp_source": flat, "x": x}], rtol=1e-30, max_iters=1)
    assert B.run(raise_on_error=False)[0]["iterations"] == 1
    B.close()
    M, S, W = (torch.from_numpy(a).to(dev) for a in line_matrices(n, 1))
    along = lambda A, v, d: torch.movedim(torch.tensordot(A, v, dims=([1], [d])), 0, d)
    b = f
    for d in range(3):
        b = along(W, b, d)
    b = b * (0.5 / n) ** 3
    kh = 1.3 * 0.5 / n
    apply = lambda v: kh * (along(M, along(M, along(S, v, 2), 1), 0) + along(M, along(S, along(M, v, 2), 1), 0)
                            + along(S, along(M, along(M, v, 2), 1), 0))
    z = b / (kh * 3 * float(S[0, 0]) * float(M[0, 0]) ** 2)    # D is one number: no node has a boundary neighbour's row
    want = z * ((b * z).sum() / (z * apply(z)).sum())
    assert float((x.view(F, F, F) - want).norm()) <= 3.2e-7 * float(want.norm())
