"""Footprints that admission reserves (host arithmetic, no GPU).  Elasticity requests do not count the
scratch of the tensor-core element matrices: an assembly without room for it uses the direct kernels,
so a server must not refuse a request for it.  The figures are those of the element matrices, the CSR,
the layouts and the solver's vectors alone."""
import pytest

from fempar_gb300 import build, serving


@pytest.mark.parametrize("kind,n,order,want", [
    (serving.ELASTICITY, (9, 8, 7), 1, (72508495, 1944)),
    (serving.ELASTICITY, (12, 12, 12), 2, (321774979, 45000)),
    (serving.ELASTICITY, (40, 40, 40), 2, (8881004180, 1574640)),
    (serving.ELASTICITY, (7, 6, 5), 3, (279234936, 19152)),
    (serving.POISSON, (12, 12, 12), 2, (105458271, 12167)),
])
def test_footprint(kind, n, order, want):
    build.build()
    assert serving.footprint(kind=kind, n=n, order=order) == want
