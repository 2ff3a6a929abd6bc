"""Cell-block (dG) CG with one slice per warp and warps that have none: the slices are not a multiple
of the warps launched (blocks = min(SMs, slices), warps rounded up per block).

* 6^3 Q2: 5,832 rows, 183 slices on 152 SMs: two warps per block, 121 without a slice.
* 9 x 8 x 7 Q1: 4,032 rows, 126 slices: one warp per block, none idle (the neighbour of the rule).
* 13 x 12 x 11 Q1: 13,728 rows, 429 slices: three warps per block, 27 idle, a last slice full.

Each solve by its true residual with the exported matrix: rtol plus the FP64 rounding of the recursive
residual (~1e-13 at these sizes, 1e-12 allowed), and the same bits twice."""
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


@pytest.mark.parametrize("n,order", [((6, 6, 6), 2), ((9, 8, 7), 1), ((13, 12, 11), 1)])
def test_warps_without_a_slice(fg, n, order):
    import scipy.sparse as sp
    ctx = fg.Context(0)
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=order, dg=True)
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(source_fn=fg.FG_FN_CONST, fn_param=[1.0],
                                                          boundary_fn=fg.FG_FN_ZERO)).compute()
    irp, ja, val = op.get_matrix(symmetric_storage=False, one_based=False)
    A = sp.csr_matrix((val, ja, irp), shape=(space.num_free_dofs,) * 2)
    b = op.get_translation()
    for prec in ("fp64", "mixed"):
        s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
        s.set_parameters_from_pl({"ILS_RTOL": 1e-10, "ILS_MAX_NUM_ITERATIONS": 20000, "PRECISION": prec})
        x = s.solve()
        assert s.info()["converged"], prec
        assert np.linalg.norm(b - A @ x) <= (1e-10 + 1e-12) * np.linalg.norm(b), prec
        assert np.array_equal(x, s.solve()), prec
    op.close()
    space.close()
    tri.close()
