"""The DCT-IV products of an inflow/outflow-x grid at the edges of their tiles (96 or 144 outputs by 64 or 128 lines,
8 terms at a time) against the oracle.  A product of N terms summed in order is within N u of the exact one (relative
L2), and a solve holds two: 5.8e-14 in FP64 and 3.1e-5 in FP32 at N = 257 if every rounding had one sign, its root
sum of squares sixteen times less; the bars are the pressure solve's, 1e-12 and 1e-5."""
import numpy as np
import pytest

from dfdm.native import Solver

from test_oracle_dct import dct_case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def oracle_mod():
    import oracle
    oracle.build()
    return oracle


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("terms", [95, 97, 143, 145, 193, 257])
@pytest.mark.parametrize("ny,nz", [(8, 10), (9, 18), (14, 12)])   # 56, 128 and 130 lines
def test_tile_edges(oracle_mod, prec, tol, terms, ny, nz):
    c = dct_case(terms + 1, ny, nz, 2)
    o = oracle_mod.Oracle(c)
    rhs = np.asfortranarray(np.random.default_rng(terms + ny).standard_normal((c.nx, ny - 1, nz)))
    want = o.solve_poisson(rhs)[:terms, :, :nz - 2]
    o.close()
    with Solver(c, prec) as s:
        got = s.solve_poisson_equation(rhs)[:terms, :, :nz - 2]
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
