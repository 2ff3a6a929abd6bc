"""BDDC where quotients leave the range in which the kernels' three-operation quotient rounds like a
division (they divide there): the FP32 apply on residuals scaled by 2^-95 and 2^95 (numerators under 2^-100,
quotients past 2^100), and an FP64 set-up whose factors' entries multiply to under 2^-960.

A power of two scales every operation exactly, up to entries that become subnormal: those are off by
at most 2^-149 per operation against values of ~2^-95 in FP32 (2^-54 of them, times the ~1,000 operations of
a row) and by 2^-1074 against 2^-960 in FP64.  Bars: one FP32 rounding, 2^-23, of the largest entry; 1e-12."""
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


def preconditioner(fg, scale):
    ctx = fg.Context(0)
    n = (6, 5, 4)
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=2, dirichlet_ids=[1, 3, 5, 7, 13, 15, 17, 19, 25])
    coef = scale * np.exp(np.random.default_rng(2).normal(size=120))
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(cell_coef=coef, source_fn=fg.FG_FN_CONST, fn_param=[1.0])).compute()
    return fg.MLBDDC(op, nsub=(2, 2, 1)), space.num_free_dofs, (ctx, tri, space, op)


def apply(fg, M, r, prec):
    import torch
    z = torch.empty_like(r)
    torch.cuda.synchronize()
    M.apply_device(r, z, prec)
    torch.cuda.synchronize()
    return z.cpu().numpy()


def test_fp32_apply_of_tiny_and_huge_residuals(fg):
    import torch
    M, n, keep = preconditioner(fg, 1.0)
    r = torch.from_numpy(np.random.default_rng(1).standard_normal(n)).cuda()
    z = apply(fg, M, r, fg.FG_MIXED)
    for e in (-95, 95):
        y = np.ldexp(apply(fg, M, r * 2.0 ** e, fg.FG_MIXED), -e)
        assert np.abs(y - z).max() <= 2.0 ** -23 * np.abs(z).max(), e
    M.close()


def test_fp64_set_up_of_a_tiny_matrix(fg):
    import torch
    M, n, keep = preconditioner(fg, 1.0)
    T, _, keep2 = preconditioner(fg, 2.0 ** -960)
    r = torch.from_numpy(np.random.default_rng(1).standard_normal(n)).cuda()
    z = apply(fg, M, r, fg.FG_FP64)
    y = apply(fg, T, r * 2.0 ** -960, fg.FG_FP64)
    assert np.abs(y - z).max() <= 1e-12 * np.abs(z).max()
    M.close()
    T.close()
