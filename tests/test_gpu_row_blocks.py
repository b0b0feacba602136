"""The x transforms with every block size their rule picks (one warp to 256 threads, from the number of x lines) and a last
block that is not full, through the pressure solve and three steps, against the oracle: FP64 1e-12, FP32 1e-5."""
import numpy as np
import pytest

from conftest import rel_l2
from dfdm import cases
from dfdm.native import Solver

pytestmark = pytest.mark.gpu

# Nx, Ny, Nz: lines = Ny Nz; threads per block 32 (few lines), 64 and 128, 256, and a length with 16-point second steps
SHAPES = [(32, 9, 8), (64, 37, 32), (64, 70, 96), (16, 150, 200), (48, 67, 256), (384, 21, 24), (512, 13, 8)]


def _channel(shape):
    return cases.channel(*shape, 3.0, 1.5, 2.0, 2000.0, 1.0, 2e-3, 41, 3, "rows")


@pytest.mark.parametrize("shape", SHAPES)
def test_pressure_solve(oracle_mod, shape):
    c = _channel(shape)
    rhs = np.asfortranarray(np.random.default_rng(3).normal(size=c.shapes()["rhs_p"]))
    n = tuple(c.cells)
    # one value per independent cell, its periodic copies equal, so that both sides solve the same field
    i, k = np.arange(rhs.shape[0]) % n[0], np.arange(rhs.shape[2]) % n[2]
    rhs = np.asfortranarray(rhs[i][:, :, k])
    o = oracle_mod.Oracle(c)
    want = o.solve_poisson(rhs)[:n[0], :n[1], :n[2]]
    for prec, tol in (("fp64", 1e-12), ("fp32", 1e-5)):
        s = Solver(c, prec)
        assert rel_l2(s.solve_poisson_equation(rhs)[:n[0], :n[1], :n[2]], want) <= tol, prec
        s.close()


@pytest.mark.parametrize("shape", SHAPES[:4])
def test_steps(oracle_mod, shape):
    c = _channel(shape)
    state = cases.initial_condition(c)
    o = oracle_mod.Oracle(c)
    o.set_state(*state)
    o.step(2)
    for prec, tol in (("fp64", 1e-12), ("fp32", 1e-5)):
        s = Solver(c, prec)
        s.set_state(*state)
        s.compute_time_step_RK3(2)
        # P is left to test_pressure_solve: phi / (0.75 dt) of a weak pressure carries the rounding of the mean flow,
        # 1e-16 u dx / dt = 4e-15 against P = 5e-3 here, times the smoothing of the solve (1e-12 to 7e-12 measured)
        for key, a, b in zip("UVW", s.get_state(), o.get_state()):
            assert rel_l2(a, b) <= tol, (prec, key)
        s.close()
