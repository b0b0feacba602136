"""The x transforms with every block size their rule picks (one warp to 256 threads, from the number of x lines), in both
orders of the spectrum (plane-major where the one-launch spectral solve runs, else row-major) and with last blocks that are
not full, through the pressure solve and two steps, against the oracle: FP64 1e-12 (the rounding of the lowest mode where the
rows are many: solve_bound), FP32 1e-5, and P at the bounds of pressure_bounds."""
import numpy as np
import pytest

from conftest import interior, pressure_bounds, rel_l2, solve_bound
from dfdm import cases
from dfdm.native import Solver

pytestmark = pytest.mark.gpu

# Nx, Ny, Nz (lines = Ny Nz): threads per block on 148 SMs, order of the spectrum, lines in a partial last block
SHAPES = [
    (32, 9, 8),       # 32, plane-major
    (64, 37, 32),     # 32, plane-major, an 8-point second step
    (64, 70, 96),     # 64, plane-major
    (16, 150, 200),   # 256, row-major, 48 of 64
    (16, 297, 24),    # 64, plane-major, 8 of 16
    (48, 311, 24),    # 128, plane-major, 8 of 16
    (384, 299, 24),   # 256, plane-major, 8 of 16, a 16-point second step
    (16, 721, 20),    # 128, row-major, 20 of 32
    (32, 199, 20),    # 32, row-major, 4 of 8
    (64, 119, 30),    # 64, row-major, 2 of 8
    (48, 67, 256),    # 256, row-major
    (384, 21, 24),    # 32, row-major, a 16-point second step
    (512, 13, 8),     # 32, row-major, a 16-point second step
]


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
    for prec, tol in (("fp64", solve_bound(c)), ("fp32", 1e-5)):
        s = Solver(c, prec)
        assert rel_l2(s.solve_poisson_equation(rhs)[:n[0], :n[1], :n[2]], want) <= tol, prec
        s.close()


@pytest.mark.parametrize("shape", SHAPES[:10])
def test_steps(oracle_mod, shape):
    c = _channel(shape)
    state = cases.initial_condition(c)
    o = oracle_mod.Oracle(c)
    o.set_state(*state)
    o.step(2)
    want = o.get_state()
    p_tol = pressure_bounds(c, oracle_mod, state, want)
    for prec, tol in (("fp64", 1e-12), ("fp32", 1e-5)):
        s = Solver(c, prec)
        s.set_state(*state)
        s.compute_time_step_RK3(2)
        got = s.get_state()
        s.close()
        for key, a, b in zip("UVW", got, want):
            assert rel_l2(a, b) <= tol, (prec, key)
        err = rel_l2(interior(c, "P", got[3]), interior(c, "P", want[3]))
        assert err <= p_tol[prec], (prec, "P", err, p_tol[prec])
