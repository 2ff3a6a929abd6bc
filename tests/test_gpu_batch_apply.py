"""The batch solver's direction-by-direction operator where it can go wrong: one cell, row blocks cut
by the mesh's end (1, 2, 4 periods of y per block), a single interior node, and rows of x too long
for the kernel's shared memory, which go in pieces (from 255 cells at order 2, 511 at order 1).

One iteration from x = 0 gives x = alpha D^-1 b, alpha = <b, D^-1 b> / <D^-1 b, A D^-1 b> (the FP32
operator), and the reported residual is ||b - A x|| / ||b|| (the float-float operator); both
against float64 products of the dense 1D matrices.  Bounds: x carries ~8 FP32 roundings per node and
those of the FP32 operator in alpha (~20 per node, averaged by the sum): 2e-6 of its norm; the
residual one FP32 rounding per node and a compensated sum: 1e-6."""
import numpy as np
import pytest

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


def line_matrices(n, p):
    """Mass, stiffness and load (node x Gauss point) of the line [-1, 1]-elements, interior nodes."""
    xq, wq = np.polynomial.legendre.leggauss(p + 1)
    nodes = np.linspace(-1.0, 1.0, p + 1)
    phi, dphi = np.zeros((p + 1, p + 1)), np.zeros((p + 1, p + 1))
    for a in range(p + 1):
        poly = np.poly1d([1.0])
        for b in range(p + 1):
            if b != a:
                poly = poly * np.poly1d([1.0, -nodes[b]]) / (nodes[a] - nodes[b])
        phi[a], dphi[a] = poly(xq), poly.deriv()(xq)
    L = p * n + 1
    M, S, W = np.zeros((L, L)), np.zeros((L, L)), np.zeros((L, n * (p + 1)))
    for c in range(n):
        i = slice(p * c, p * c + p + 1)
        M[i, i] += (phi * wq) @ phi.T
        S[i, i] += (dphi * wq) @ dphi.T
        W[i, c * (p + 1):(c + 1) * (p + 1)] += phi * wq
    return M[1:-1, 1:-1], S[1:-1, 1:-1], W[1:-1]


@pytest.mark.parametrize("n,p", [(2, 1), (1, 2), (1, 3), (7, 1), (5, 2), (3, 3), (13, 3), (511, 1), (256, 2)])
def test_one_iteration(env, n, p):
    ctx, torch = env
    from fempar_gb300.batch import BatchSolver
    F = p * n - 1
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev)
    g.manual_seed(n + p)
    f = torch.randn(n ** 3 * (p + 1) ** 3, dtype=torch.float64, device=dev, generator=g)
    x = torch.zeros(F ** 3, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()  # the solver has its own stream
    B = BatchSolver(ctx, [{"n": n, "order": p, "coef": 1.7, "qp_source": f, "x": x}], rtol=1e-30, max_iters=1,
                    threads=256)
    res = B.run(raise_on_error=False)[0]
    assert res["iterations"] == 1
    B.close()
    M, S, W = (torch.from_numpy(a).to(dev) for a in line_matrices(n, p))

    def along(A, v, d):  # A on direction d of v[z][y][x]
        return torch.movedim(torch.tensordot(A, v, dims=([1], [d])), 0, d)

    q = p + 1
    b = f.view(n, n, n, q, q, q).permute(0, 3, 1, 4, 2, 5).reshape(n * q, n * q, n * q)
    for d in range(3):
        b = along(W, b, d)
    b = b * (0.5 / n) ** 3
    kh = 1.7 * 0.5 / n
    apply = lambda v: kh * (along(M, along(M, along(S, v, 2), 1), 0) + along(M, along(S, along(M, v, 2), 1), 0)
                            + along(S, along(M, along(M, v, 2), 1), 0))
    m, s = torch.diag(M), torch.diag(S)
    diag = kh * (m[:, None, None] * m[:, None] * s + m[:, None, None] * s[:, None] * m
                 + s[:, None, None] * m[:, None] * m)
    z = b / diag
    want = z * ((b * z).sum() / (z * apply(z)).sum())
    x = x.view(F, F, F)
    assert float((x - want).norm()) <= 2e-6 * float(want.norm())
    rel = float((b - apply(x)).norm() / b.norm())
    assert abs(res["rel_residual"] - rel) <= 1e-6 * max(rel, 1e-6)
