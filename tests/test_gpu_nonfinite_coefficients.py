"""NaN and infinite cell coefficients: the tensor-core element matrices are non-finite exactly where
the FP64-pipe kernels' are (FG_TC_INTEGRATION=0), and every finite entry is a finite entry of theirs:
elasticity Q2 and Q3, Poisson Q1 (above 4096 cells) to Q3, the dG volume terms.  The dense product
gives non-finite rows and columns of C where A and B have them, and leaves the others alone."""
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


@pytest.fixture(scope="module")
def ctx(fg):
    return fg.Context(0)


@pytest.mark.parametrize("kind,n,order", [("elasticity", (4, 3, 3), 2), ("elasticity", (3, 3, 2), 3),
                                          ("poisson", (17, 17, 16), 1), ("poisson", (4, 4, 3), 2),
                                          ("poisson", (3, 3, 3), 3), ("dg", (3, 4, 2), 2)])
def test_matrix_and_load_keep_nonfinite_cells(fg, ctx, monkeypatch, kind, n, order):
    rng = np.random.default_rng(order)
    coef = np.exp(rng.normal(size=int(np.prod(n))))
    bad = coef.copy()
    bad[1] = np.nan
    bad[-2] = np.inf
    tri = fg.SerialTriangulation(ctx, n)
    if kind == "dg":
        space = fg.SerialFESpace(tri, order=order, dg=True)
    else:
        space = fg.SerialFESpace(tri, order=order, ncomp=3 if kind == "elasticity" else 1, dirichlet_ids=[1, 3, 5, 7])
    out = {}
    for tc in ("0", "2"):
        monkeypatch.setenv("FG_TC_INTEGRATION", tc)
        if kind == "elasticity":
            integ = fg.ElasticityIntegration(cell_coef=bad, nu=0.3, source_fn=fg.FG_FN_CONST, fn_param=[0.0, 1.0, -1.0])
        else:
            integ = fg.PoissonIntegration(cell_coef=bad, source_fn=fg.FG_FN_CONST, fn_param=[1.0])
        op = fg.FEAffineOperator(space, integ)
        try:
            op.compute()
        except fg.FGError:
            out[tc] = None  # refused (then on both paths)
            continue
        out[tc] = op.get_matrix(symmetric_storage=False, one_based=False)[2], op.get_translation()
        op.close()
    assert (out["0"] is None) == (out["2"] is None)
    if out["0"] is not None:
        for a, b in zip(out["0"], out["2"]):
            assert np.array_equal(np.isfinite(a), np.isfinite(b))
        assert not np.isfinite(out["2"][0]).all()
    space.close()
    tri.close()


@pytest.mark.parametrize("m,n,k", [(130, 70, 33), (257, 300, 200)])
@pytest.mark.parametrize("order", ["row", "column"])
def test_dense_product(fg, ctx, m, n, k, order):
    import torch
    from fempar_gb300.dense import gemm_nt
    g = torch.Generator(device="cuda").manual_seed(m)
    A = torch.randn(m, k, dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn(n, k, dtype=torch.float64, device="cuda", generator=g)
    A[3, 5] = float("nan")
    A[m - 1, 0] = float("inf")
    B[n - 2, k - 1] = float("-inf")
    C = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    if order == "column":
        C = torch.zeros(n, m, dtype=torch.float64, device="cuda").t()
    torch.cuda.synchronize()
    gemm_nt(ctx, A, B, C)
    bad = torch.zeros(m, n, dtype=torch.bool, device="cuda")
    bad[3] = bad[m - 1] = True
    bad[:, n - 2] = True
    assert torch.equal(~torch.isfinite(C), bad)
    ok = A.clone()
    ok[3] = ok[m - 1] = 0.0
    bk = B.clone()
    bk[n - 2] = 0.0
    want = ok @ bk.t()
    scale = A.abs().nan_to_num(posinf=0.0).amax(1)[:, None] * B.abs().nan_to_num(posinf=0.0).amax(1)[None]
    err = ((C - want).abs() / scale)[~bad].max().item()
    assert err <= k * 2.0 ** -52
