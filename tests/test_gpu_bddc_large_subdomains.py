"""BDDC with few, large subdomains: the apply's triangular solves keep a subdomain's vector and a 32 x 32
tile pair in shared memory (past 48 KB together from ~3,600 dofs in FP64, 9,900 in FP32), and walk 32
rows at a time (ragged last steps).  Solutions against Jacobi-PCG in FP64 on the same system: both stop
at 1e-12 of the right-hand side, and 1e-9 of the solution leaves three decades for the condition
number of these small boxes (all faces fixed)."""
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


@pytest.mark.parametrize("n,nsub,order", [((10, 5, 5), (2, 1, 1), 2), ((14, 7, 7), (2, 1, 1), 2),
                                          ((5, 4, 3), (2, 2, 1), 2), ((4, 3, 2), (2, 1, 1), 1)])
def test_solution(fg, n, nsub, order):
    ctx = fg.Context(0)
    rng = np.random.default_rng(sum(n))
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=order, ncomp=3, dirichlet_ids=list(range(1, 27)))
    coef = np.exp(0.5 * rng.normal(size=n[0] * n[1] * n[2]))
    op = fg.FEAffineOperator(space, fg.ElasticityIntegration(cell_coef=coef, nu=0.3, source_fn=fg.FG_FN_CONST,
                                                             fn_param=[0.0, 0.0, -1.0])).compute()
    ref = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
    ref.set_parameters_from_pl({"ILS_RTOL": 1e-12, "ILS_MAX_NUM_ITERATIONS": 20000})
    x = ref.solve()
    M = fg.MLBDDC(op, nsub=nsub)
    for kind, rtol in (("CG", 1e-12), ("GPU_MPCG", 1e-12)):
        s = fg.IterativeLinearSolver().set_type_from_string(kind).set_operators(op, M)
        s.set_parameters_from_pl({"ILS_RTOL": rtol, "ILS_MAX_NUM_ITERATIONS": 2000})
        y = s.solve()
        assert s.info()["converged"], kind
        assert np.linalg.norm(y - x) <= 1e-9 * np.linalg.norm(x), kind
    M.close()
