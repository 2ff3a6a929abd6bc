"""FG_PCG_BARRIER_TIMEOUT_MS: values that are not a positive number of milliseconds leave the default
bound of 10 s in place.  Solves on many blocks succeed with such values, and where a block skips its
first arrival (the bounded wait runs out) the solve fails after the bound in force: 200 ms, or the
default (not at once, which a value read as 0 ms gives)."""
import time
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


def test_values_that_are_no_limit(fg, monkeypatch):
    ctx = fg.Context(0)
    tri = fg.SerialTriangulation(ctx, (40, 40, 40))
    space = fg.SerialFESpace(tri, order=2, dirichlet_ids=list(range(1, 27)))
    op = fg.FEAffineOperator(space, fg.PoissonIntegration(source_fn=fg.FG_FN_CONST, fn_param=[1.0])).compute()
    s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
    s.set_parameters_from_pl({"ILS_RTOL": 1e-8, "ILS_MAX_NUM_ITERATIONS": 5000})
    x = s.solve()
    for value in ("0", "-5", "abc", "", "0ms", "1e400"):
        monkeypatch.setenv("FG_PCG_BARRIER_TIMEOUT_MS", value)
        assert np.array_equal(x, s.solve()), value
    monkeypatch.setenv("FG_PCG_BARRIER_TIMEOUT_MS", "200")
    assert np.array_equal(x, s.solve())
    monkeypatch.setenv("FG_PCG_TEST_DROP_ARRIVAL", "1")
    for value, least, most in (("200", 0.2, 5.0), ("0", 9.0, 30.0)):
        monkeypatch.setenv("FG_PCG_BARRIER_TIMEOUT_MS", value)
        t0 = time.perf_counter()
        with pytest.raises(fg.FGError) as e:
            s.solve()
        assert e.value.status == -6
        assert least <= time.perf_counter() - t0 <= most, value
