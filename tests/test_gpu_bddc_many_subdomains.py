"""BDDC's FP32 apply on more small subdomains than twice the SMs (343 and 512 of 2^3 cells: the kernels with
room for four CTAs per SM) and on fewer (64): against the FP64 apply of the same preconditioner.  Bar: FP32
factors and vectors, cond(A) 2^-24 with the small boxes' condition numbers of ~1e2: 1e-4 of the norm;
and solves by their true residual."""
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


@pytest.mark.parametrize("nsub,order", [(4, 2), (7, 1), (7, 2), (8, 1)])
def test_apply_and_solve(fg, nsub, order):
    import scipy.sparse as sp
    import torch
    ctx = fg.Context(0)
    n = (2 * nsub,) * 3
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=order, dirichlet_ids=list(range(1, 27)))
    coef = np.exp(0.5 * np.random.default_rng(nsub).normal(size=n[0] ** 3))
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(cell_coef=coef, source_fn=fg.FG_FN_CONST, fn_param=[1.0])).compute()
    M = fg.MLBDDC(op, nsub=(nsub,) * 3)
    r = torch.from_numpy(np.random.default_rng(1).standard_normal(space.num_free_dofs)).cuda()
    z = {}
    for prec in (fg.FG_FP64, fg.FG_MIXED):
        z[prec] = torch.empty_like(r)
        torch.cuda.synchronize()
        M.apply_device(r, z[prec], prec)
        torch.cuda.synchronize()
    assert float((z[fg.FG_MIXED] - z[fg.FG_FP64]).norm()) <= 1e-4 * float(z[fg.FG_FP64].norm())
    irp, ja, val = op.get_matrix(symmetric_storage=False, one_based=False)
    A = sp.csr_matrix((val, ja, irp), shape=(space.num_free_dofs,) * 2)
    b = op.get_translation()
    s = fg.IterativeLinearSolver().set_type_from_string("GPU_MPCG").set_operators(op, M)
    s.set_parameters_from_pl({"ILS_RTOL": 1e-10, "ILS_MAX_NUM_ITERATIONS": 500})
    x = s.solve()
    assert s.info()["converged"]
    assert np.linalg.norm(b - A @ x) <= (1e-10 + 1e-12) * np.linalg.norm(b)
    M.close()
