"""Streaming CG launches of half the width, whose blocks do two of the solve's each (what a server uses
while other requests solve; FG_PCG_TEST_SHARE=1 forces it): the same bits as full launches, for every
streaming kernel (both precisions, the three layouts, FP64 explicit columns past 170 MB), all reductions
(with and without preconditioner, a criterion on the step) and short launches.  And a server's concurrent
streaming solves equal a single worker's."""
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


@pytest.mark.parametrize("kind,n,order,layout", [("poisson", (69, 69, 69), 1, "stencil"), ("elasticity", (19, 19, 19), 2, "stencil"),
                                                 ("poisson", (69, 69, 69), 1, "sell"), ("poisson", (38, 36, 37), 2, "sell"),
                                                 ("dg", (34, 34, 34), 1, "dg")])
def test_same_bits(fg, monkeypatch, kind, n, order, layout):
    if layout == "sell":
        monkeypatch.setenv("FG_SOLVER_LAYOUT", "sell")
    ctx = fg.Context(0)
    tri = fg.SerialTriangulation(ctx, n)
    coef = np.exp(np.random.default_rng(1).normal(size=int(np.prod(n))))
    if kind == "dg":
        space = fg.SerialFESpace(tri, order=order, dg=True)
        integ = fg.PoissonIntegration(source_fn=fg.FG_FN_CONST, fn_param=[1.0])
    elif kind == "elasticity":
        space = fg.SerialFESpace(tri, order=order, ncomp=3, dirichlet_ids=[1, 3, 5, 7, 13, 15, 17, 19, 25])
        integ = fg.ElasticityIntegration(cell_coef=coef, nu=0.3, source_fn=fg.FG_FN_CONST, fn_param=[0.0, 0.0, -1.0])
    else:
        space = fg.SerialFESpace(tri, order=order, dirichlet_ids=list(range(1, 27)))
        integ = fg.PoissonIntegration(cell_coef=coef, source_fn=fg.FG_FN_CONST, fn_param=[1.0])
    op = fg.FEAffineOperator(space, integ).compute()
    for prec, precond, extra in (("fp64", "jacobi", {}), ("fp64", "identity", {}), ("mixed", "jacobi", {}),
                                 ("fp64", "jacobi", {"ILS_STOPPING_CRITERIUM": "delta_delta"}),
                                 ("mixed", "identity", {}), ("mixed", "jacobi", {"CHECK_EVERY": 5})):
        s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, precond)
        s.set_parameters_from_pl({"ILS_RTOL": 1e-7, "ILS_MAX_NUM_ITERATIONS": 120, "PRECISION": prec, **extra})
        x, i = s.solve(), s.info()["iterations"]
        monkeypatch.setenv("FG_PCG_TEST_SHARE", "1")
        assert np.array_equal(x, s.solve()) and s.info()["iterations"] == i, (prec, precond, extra)
        monkeypatch.delenv("FG_PCG_TEST_SHARE")
    op.close()
    space.close()
    tri.close()


def test_server_gives_the_same_bits_alone_and_beside_others(fg):
    from fempar_gb300 import serving
    rng = np.random.default_rng(4)
    reqs = [dict(kind=serving.ELASTICITY, n=(19, 19, 19), order=2, cell_coef=np.exp(rng.normal(size=19 ** 3)), rtol=1e-5),
            dict(kind=serving.POISSON, n=(70, 69, 69), order=1, cell_coef=np.exp(rng.normal(size=70 * 69 * 69)),
                 precision=fg.FG_FP64, rtol=1e-8),
            dict(kind=serving.POISSON, n=(44, 44, 44), order=2, cell_coef=np.exp(rng.normal(size=44 ** 3))),
            dict(kind=serving.POISSON, n=(12, 12, 12), order=2, cell_coef=np.exp(rng.normal(size=12 ** 3)))]
    out = []
    for workers in (1, 4):
        srv = serving.Server(nworkers=workers)
        tickets = [srv.submit(**rq) for _ in range(2) for rq in reqs]
        xs = []
        for t in tickets:
            r = srv.wait(t)
            assert r["status"] == 0
            xs.append(srv.take(t, r["num_free"]))
        srv.close()
        out.append(xs)
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind,n,order", [("poisson", (9, 8, 7), 2), ("poisson", (26, 24, 25), 2), ("poisson", (40, 36, 38), 2),
                                          ("elasticity", (19, 19, 19), 2)],
                         ids=["one_block", "one_slice_per_warp", "two_slices_per_warp", "streamed"])
def test_bits_do_not_depend_on_the_length_of_launches(fg, monkeypatch, kind, n, order):
    """Launches of 1, 3, 8 and 21 iterations against the default (~5 ms): the stop estimate of the mixed
    iteration is taken at the same iterations of a segment whatever launch they are in."""
    ctx = fg.Context(0)
    tri = fg.SerialTriangulation(ctx, n)
    coef = np.exp(np.random.default_rng(1).normal(size=int(np.prod(n))))
    if kind == "elasticity":
        space = fg.SerialFESpace(tri, order=order, ncomp=3, dirichlet_ids=[1, 3, 5, 7, 13, 15, 17, 19, 25])
        integ = fg.ElasticityIntegration(cell_coef=coef, nu=0.3, source_fn=fg.FG_FN_CONST, fn_param=[0.0, 0.0, -1.0])
    else:
        space = fg.SerialFESpace(tri, order=order, dirichlet_ids=list(range(1, 27)))
        integ = fg.PoissonIntegration(cell_coef=coef, source_fn=fg.FG_FN_CONST, fn_param=[1.0])
    op = fg.FEAffineOperator(space, integ).compute()
    for prec in ("mixed", "fp64"):
        s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
        s.set_parameters_from_pl({"ILS_RTOL": 1e-5, "ILS_MAX_NUM_ITERATIONS": 5000, "PRECISION": prec})
        x, i = s.solve(), s.info()["iterations"]
        assert s.info()["converged"]
        for its in ("1", "3", "8", "21"):
            monkeypatch.setenv("FG_PCG_TEST_LAUNCH_ITERS", its)
            assert np.array_equal(x, s.solve()) and s.info()["iterations"] == i, (prec, its)
        monkeypatch.delenv("FG_PCG_TEST_LAUNCH_ITERS")
    op.close()
    space.close()
    tri.close()
