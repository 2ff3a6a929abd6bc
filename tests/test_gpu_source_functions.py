"""Every source function on every integration path, with parameters that only some of them read (the
boundary function shares fn_param): right-hand sides against the oracle's.  FG_FN_LINEAR and FG_FN_ZERO
are f = 0 whatever fn_param holds.

Paths: FG_TC_INTEGRATION 0 (FP64 pipe), 2 (tensor cores; Q1 above 4096 cells too), and a fast request
(float-float geometry); continuous and dG.  Bars: 1e-13 of the largest entry, 1e-12 for fast requests
(the float-float geometry's bar)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
SHARP = [25.0, 0.3, -0.05, -0.05, -0.05]
SOURCES = [O.FN_ZERO, O.FN_CONST, O.FN_SHARP_WAVE, O.FN_LINEAR, O.FN_QP_VALUES]


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


@pytest.mark.parametrize("n,order,dg", [((4, 3, 2), 1, False), ((17, 17, 16), 1, False), ((4, 3, 5), 2, False),
                                        ((3, 2, 3), 3, False), ((4, 3, 2), 1, True), ((17, 17, 16), 1, True),
                                        ((3, 4, 2), 2, True), ((2, 3, 2), 3, True)])
def test_right_hand_sides(fg, ctx, n, order, dg, monkeypatch):
    rng = np.random.default_rng(order + sum(n))
    nqp = int(np.prod(n)) * (order + 1) ** 3
    qp = rng.standard_normal(nqp)
    tri = fg.SerialTriangulation(ctx, n)
    ids = [] if dg else list(range(1, 27))
    space = fg.SerialFESpace(tri, order=order, dg=True) if dg else fg.SerialFESpace(tri, order=order, dirichlet_ids=ids)
    for fn in SOURCES:
        src = {"source_fn": fn, "boundary_fn": O.FN_CONST, "fn_param": SHARP}
        if fn == O.FN_QP_VALUES:
            src["qp_source"] = qp
        P = O.Problem(n, order=order, formulation=O.DG if dg else O.CG, **src)
        want = P.rhs()
        for tc, fast in (("0", False), ("2", False), ("2", True)):
            monkeypatch.setenv("FG_TC_INTEGRATION", tc)
            op = fg.FEAffineOperator(space, fg.PoissonIntegration(fast_integration=fast, **src)).compute()
            got = op.get_translation()
            tol = 1e-12 if fast else 1e-13
            assert np.abs(got - want).max() <= tol * max(np.abs(want).max(), 1e-300), (fn, tc, fast)
            op.close()
    space.close()
    tri.close()
