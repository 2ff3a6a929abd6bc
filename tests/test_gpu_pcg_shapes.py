"""The cooperative CG kernels at the edges of their launch shapes: one block, one slice per warp,
two slices per warp, streamed vectors; both matrix layouts, FP64 and mixed precision.

Each solve is checked by its true residual with the exported matrix (the recursive residual of
CG in FP64 stays within rounding, ~1e-13 of the right-hand side at these sizes, of the true one)
and, at the small sizes, against the oracle's iteration counts (+-1)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu

# cells per direction (Q1, interior nodes free) -> slices of 32 rows on 152 SMs
SHAPES = [
    ((2, 2, 2), "one row"),
    ((9, 9, 9), "16 slices: the last single block"),
    ((9, 9, 10), "18 slices: more than one block"),
    ((25, 30, 23), "479 slices: a warp or two per SM's block"),
    ((54, 55, 54), "4740 slices: one per warp, below 4864"),
    ((55, 55, 55), "4921 slices: two per warp"),
    ((69, 68, 69), "9682 slices: two per warp, below 9728"),
    ((69, 69, 69), "9826 slices: streamed"),
]


@pytest.fixture(scope="module")
def fg():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fempar_gb300 as fg
    from fempar_gb300 import build
    build.build()
    return fg


@pytest.fixture(scope="module")
def ctx(fg):
    return fg.Context(0)


@pytest.mark.parametrize("layout", ["stencil", "sell"])
@pytest.mark.parametrize("n", [s[0] for s in SHAPES], ids=[s[1].split(":")[0].replace(" ", "_") for s in SHAPES])
def test_pcg_shapes(fg, ctx, n, layout, monkeypatch):
    import scipy.sparse as sp
    if layout == "sell":
        monkeypatch.setenv("FG_SOLVER_LAYOUT", "sell")
    rng = np.random.default_rng(sum(n))
    coef = np.exp(rng.normal(size=n[0] * n[1] * n[2]))
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=1, dirichlet_ids=list(range(1, 27)))
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(cell_coef=coef, source_fn=fg.FG_FN_CONST,
                                                          fn_param=[1.0])).compute()
    irp, ja, val = op.get_matrix(symmetric_storage=False, one_based=False)
    A = sp.csr_matrix((val, ja, irp), shape=(space.num_free_dofs,) * 2)
    b = op.get_translation()
    nb = np.linalg.norm(b)
    for prec, precond, rtol in (("fp64", "jacobi", 1e-11), ("fp64", "identity", 1e-9), ("mixed", "jacobi", 1e-11)):
        s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, precond)
        s.set_parameters_from_pl({"ILS_RTOL": rtol, "ILS_MAX_NUM_ITERATIONS": 20000, "PRECISION": prec})
        x = s.solve()
        assert s.info()["converged"], (prec, precond)
        assert np.linalg.norm(b - A @ x) <= (rtol + 1e-12) * nb, (prec, precond)
        x2 = s.solve()
        assert np.array_equal(x, x2), "not deterministic"
        if prec == "fp64" and space.num_free_dofs < 20000:
            P = O.Problem(n, order=1, cell_coef=coef, source_fn=O.FN_CONST, fn_param=[1.0])
            # the oracle's own count moves with its summation order (one thread, four, full rows): 147,
            # 145 and 147 without a preconditioner on 25 x 30 x 23
            its = [P.cg(precond=int(precond == "jacobi"), rtol=rtol, maxit=20000, nthreads=t)["iters"]
                   for t in (1, 4, -4)]
            assert min(its) - 1 <= s.info()["iterations"] <= max(its) + 1
    # a launch per few iterations gives the same solution as long launches
    s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
    s.set_parameters_from_pl({"ILS_RTOL": 1e-11, "ILS_MAX_NUM_ITERATIONS": 20000})
    x = s.solve()
    s.set_parameters_from_pl({"CHECK_EVERY": 7})
    assert np.array_equal(x, s.solve())
    op.close()
    space.close()
    tri.close()


@pytest.mark.parametrize("n,order", [((1, 1, 1), 1), ((5, 3, 2), 2), ((2, 3, 2), 3), ((30, 30, 30), 1), ((34, 34, 34), 1)],
                         ids=["one_cell", "ragged_slice", "q3", "two_slices_per_warp", "streamed"])
def test_dg_cell_block_layout(fg, ctx, n, order):
    """The dG layout whose columns follow from the cell and its neighbours: products with the
    exported CSR (FP64 and FP32), and solves by their true residual, at the edges of the shapes."""
    import scipy.sparse as sp
    import torch
    rng = np.random.default_rng(order + sum(n))
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=order, dg=True)
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(source_fn=fg.FG_FN_CONST, fn_param=[1.0],
                                                          boundary_fn=fg.FG_FN_ZERO)).compute()
    irp, ja, val = op.get_matrix(symmetric_storage=False, one_based=False)
    A = sp.csr_matrix((val, ja, irp), shape=(space.num_free_dofs,) * 2)
    x = rng.standard_normal(space.num_free_dofs)
    scale = abs(A) @ abs(x)
    m = np.diff(irp).max()
    for prec, dt, eps in ((fg.FG_FP64, torch.float64, 2.0 ** -53), (fg.FG_MIXED, torch.float32, 2.0 ** -24)):
        dx = torch.from_numpy(x).to("cuda", dt)
        y = op.apply_device(dx, torch.empty_like(dx), prec).double().cpu().numpy()
        # m products summed, and the roundings of the values and of x to the type
        assert np.all(np.abs(y - A @ x) <= (m + 3) * eps * scale)
    b = op.get_translation()
    for prec in ("fp64", "mixed"):
        s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
        s.set_parameters_from_pl({"ILS_RTOL": 1e-10, "ILS_MAX_NUM_ITERATIONS": 20000, "PRECISION": prec})
        x = s.solve()
        assert s.info()["converged"], prec
        assert np.linalg.norm(b - A @ x) <= (1e-10 + 1e-12) * np.linalg.norm(b), prec
    op.close()
    space.close()
    tri.close()


def test_pcg_bounded_barrier_runs_out_and_context_survives(fg, ctx, monkeypatch):
    """A block that skips its first arrival: the bounded grid barriers run out, the solve reports
    FG_ERR_TIMEOUT and the same system then solves."""
    n = (12, 11, 10)
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=1, dirichlet_ids=list(range(1, 27)))
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(source_fn=fg.FG_FN_CONST, fn_param=[1.0])).compute()
    s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
    for prec in ("fp64", "mixed"):
        s.set_parameters_from_pl({"ILS_RTOL": 1e-10, "PRECISION": prec})
        monkeypatch.setenv("FG_PCG_TEST_DROP_ARRIVAL", "1")
        monkeypatch.setenv("FG_PCG_BARRIER_TIMEOUT_MS", "200")
        with pytest.raises(fg.FGError) as e:
            s.solve()
        assert e.value.status == -6
        monkeypatch.delenv("FG_PCG_TEST_DROP_ARRIVAL")
        monkeypatch.delenv("FG_PCG_BARRIER_TIMEOUT_MS")
        s.solve()
        assert s.info()["converged"]


@pytest.mark.parametrize("n,order,layout", [((5, 4, 3), 3, "stencil"), ((13, 12, 11), 3, "stencil"),
                                            ((13, 12, 11), 3, "sell"), ((20, 17, 19), 2, "sell"),
                                            ((38, 36, 37), 2, "sell")])
def test_slices_kept_in_shared_memory(fg, ctx, n, order, layout, monkeypatch):
    """Matrices of which a block holds all its slices in shared memory, or the first ones that fit (42
    MB of FP64 values on 152 SMs), slices of every width, and one streamed from HBM (203 MB of FP64
    values with columns beside them): solves by their true residual."""
    import scipy.sparse as sp
    if layout == "sell":
        monkeypatch.setenv("FG_SOLVER_LAYOUT", "sell")
    rng = np.random.default_rng(order + sum(n))
    coef = np.exp(rng.normal(size=n[0] * n[1] * n[2]))
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=order, dirichlet_ids=list(range(1, 27)))
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(cell_coef=coef, source_fn=fg.FG_FN_CONST,
                                                          fn_param=[1.0])).compute()
    irp, ja, val = op.get_matrix(symmetric_storage=False, one_based=False)
    A = sp.csr_matrix((val, ja, irp), shape=(space.num_free_dofs,) * 2)
    b = op.get_translation()
    for prec in ("fp64", "mixed"):
        s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
        s.set_parameters_from_pl({"ILS_RTOL": 1e-10, "ILS_MAX_NUM_ITERATIONS": 20000, "PRECISION": prec})
        x = s.solve()
        assert s.info()["converged"], prec
        assert np.linalg.norm(b - A @ x) <= (1e-10 + 1e-12) * np.linalg.norm(b), prec
        assert np.array_equal(x, s.solve()), "not deterministic"
    op.close()
    space.close()
    tri.close()
