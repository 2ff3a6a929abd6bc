"""A CG iteration that overflows inside the last polling chunk before the iteration limit: the solve runs
to the limit and reports that it did not converge; it is an error only where a chunk ends before the
limit.  The polling chunk is 64 iterations below 200,000 dofs.

13^3 Q3 elasticity, 164,502 dofs, ~62 M matrix entries: a launch takes fewer iterations than a chunk.
The right-hand side is scaled to <b,b> = 1.4e308, so the first growth of the residual by 12 % overflows
(no preconditioner and lognormal coefficients: within a few iterations; the matrix entries are ~1e-9, so
<p,Ap> does not)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import fempar_gb300 as fg
    from fempar_gb300 import build
    build.build()
    ctx = fg.Context(0)
    n = (13, 13, 13)
    coef = 1e-9 * np.exp(np.random.default_rng(1).normal(size=13 ** 3))
    tri = fg.SerialTriangulation(ctx, n)
    space = fg.SerialFESpace(tri, order=3, ncomp=3, dirichlet_ids=[1, 3, 5, 7, 13, 15, 17, 19, 25])
    assert space.num_free_dofs < 200000
    op = fg.FEAffineOperator(space, fg.ElasticityIntegration(cell_coef=coef, nu=0.3, source_fn=fg.FG_FN_CONST,
                                                             fn_param=[0.0, 0.0, -1.0])).compute()
    b = op.get_translation()
    return fg, op, b * (1.2e154 / np.linalg.norm(b)), (tri, space, ctx)


@pytest.mark.parametrize("limit,error", [(5, False), (60, False), (64, False), (65, True), (200, True)])
def test_overflow(system, limit, error):
    fg, op, b, _ = system
    s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "identity")
    s.set_parameters_from_pl({"ILS_RTOL": 1e-10, "ILS_MAX_NUM_ITERATIONS": limit, "PRECISION": "fp64"})
    if error:
        with pytest.raises(fg.FGError) as e:
            s.solve(b)
        assert e.value.status == -5
    else:
        x = s.solve(b)
        assert s.info()["iterations"] == limit and not s.info()["converged"]
        if limit == 60:
            assert not np.isfinite(x).all(), "the case did not overflow"
