"""The scratch of the tensor-core element matrices (elasticity, dG) and the HBM budget: it is taken only
where there is room, and given back when the element matrices are done.

* A budget that an assembly on the FP64-pipe kernels and the solve after it just fit in: the default
  path assembles and solves in it too (1 MiB more: the shared tables, 0.74 MB for Q2).
* A full system holds no more after its assembly than one assembled on the FP64 pipe, the tables
  aside, and so again after a reassembly.
* A server whose budget is one elasticity request's footprint serves it, and keeps to the budget."""
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


def problem(fg, ctx, kind):
    n = (6, 5, 4) if kind == "elasticity" else (8, 8, 7)
    coef = np.exp(np.random.default_rng(3).normal(size=int(np.prod(n))))
    tri = fg.SerialTriangulation(ctx, n)
    if kind == "elasticity":
        space = fg.SerialFESpace(tri, order=2, ncomp=3, dirichlet_ids=[1, 3, 5, 7, 13, 15, 17, 19, 25])
        integ = fg.ElasticityIntegration(cell_coef=coef, nu=0.3, source_fn=fg.FG_FN_CONST, fn_param=[0.0, 0.0, -1.0])
    else:
        space = fg.SerialFESpace(tri, order=2, dg=True)
        integ = fg.PoissonIntegration(source_fn=fg.FG_FN_CONST, fn_param=[1.0])
    return tri, space, fg.FEAffineOperator(space, integ)


def solve(fg, op):
    s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
    s.set_parameters_from_pl({"ILS_RTOL": 1e-8, "ILS_MAX_NUM_ITERATIONS": 20000, "PRECISION": "mixed"})
    x = s.solve()
    assert s.info()["converged"]
    return x


@pytest.mark.parametrize("kind", ["elasticity", "dg"])
def test_budget_of_the_direct_kernels_is_enough(fg, monkeypatch, kind):
    monkeypatch.setenv("FG_TC_INTEGRATION", "0")
    ca = fg.Context(0)
    keep = problem(fg, ca, kind)
    keep[2].compute()
    x = solve(fg, keep[2])
    budget = ca.memory()[0] + (1 << 20)
    monkeypatch.delenv("FG_TC_INTEGRATION")
    cb = fg.Context(0, hbm_budget_bytes=budget)
    keep2 = problem(fg, cb, kind)
    keep2[2].compute()
    y = solve(fg, keep2[2])
    # two solves to 1e-8 of the residual on matrices that agree to ~1e-14: the condition number is ~1e4
    assert np.linalg.norm(x - y) <= 1e-4 * np.linalg.norm(x)


@pytest.mark.parametrize("kind", ["elasticity", "dg"])
def test_scratch_is_given_back(fg, monkeypatch, kind):
    used = {}
    for tc in ("0", "2"):
        monkeypatch.setenv("FG_TC_INTEGRATION", tc)
        ctx = fg.Context(0)
        keep = problem(fg, ctx, kind)
        keep[2].compute()
        used[tc] = ctx.memory()[0]
        keep[2].compute()
        assert ctx.memory()[0] == used[tc]
    assert used["2"] <= used["0"] + (1 << 20)


def test_server_with_one_request_of_budget(fg):
    from fempar_gb300 import serving
    rq = dict(kind=serving.ELASTICITY, n=(12, 12, 12), order=2)
    need, nfree = serving.footprint(**rq)
    xs = []
    for budget in (need, 8 << 30):
        srv = serving.Server(hbm_budget_bytes=budget, nworkers=2)
        tickets = [srv.submit(**rq) for _ in range(2)]
        for t in tickets:
            r = srv.wait(t)
            assert r["status"] == 0 and r["num_free"] == nfree
            xs.append(srv.take(t, nfree))
        assert srv.stats()["peak_reserved_bytes"] <= budget
        srv.close()
    for x in xs[1:]:
        assert np.linalg.norm(x - xs[0]) <= 1e-4 * np.linalg.norm(xs[0])
