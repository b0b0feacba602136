"""The one-launch spectral solve of wall-bounded grids (k_plane: z transforms and tridiagonal solves of a kx plane in a pair
of blocks) where its rule takes it and next to where it does not, against the oracle: the pressure solve and two steps, FP64
1e-12, FP32 1e-5 relative L2, P after the steps at the bounds of pressure_bounds; the launch count of a step tells which path
ran (13 kernels with it, 19 without)."""
import numpy as np
import pytest

from conftest import interior, pressure_bounds, rel_l2
from dfdm import cases
from dfdm.native import Solver

pytestmark = pytest.mark.gpu

# shape, FP64 takes it, FP32 takes it
SHAPES = [
    ((16, 3, 8), True, True),          # the fewest rows: two and one
    ((16, 4, 24), True, True),
    ((32, 47, 48), True, True),        # halves of 24 and 23 rows
    ((96, 21, 32), True, True),        # small planes, up to 49 of them
    ((128, 21, 32), False, False),     # ... and more
    ((128, 48, 48), True, True),       # from 48 x 48 cells
    ((16, 146, 128), True, True),      # the largest half plane of FP64
    ((16, 150, 128), False, True),
    ((64, 110, 256), False, True),     # the largest of FP32
    ((64, 112, 256), False, False),
    ((32, 30, 256), False, False),     # Nz = 256 with few planes
    ((64, 30, 192), True, True),
    ((20, 30, 32), False, False),      # Nx/2 = 10 has no two-level split
]


@pytest.mark.parametrize("shape,fp64,fp32", SHAPES, ids=["x".join(map(str, s[0])) for s in SHAPES])
def test_against_the_oracle(oracle_mod, shape, fp64, fp32):
    c = cases.channel(*shape, 3.0, 1.5, 2.0, 2000.0, 1.0, 2e-3, 43, 2, "plane").with_(flow_forcing_mode=0, dPdx=1.0)
    state = cases.initial_condition(c)
    o = oracle_mod.Oracle(c)
    o.set_state(*state)
    rhs = o.divergence_rhs()
    n = tuple(c.cells)
    phi = o.solve_poisson(rhs)[:n[0], :n[1], :n[2]]
    o.step(2)
    want = o.get_state()
    p_tol = pressure_bounds(c, oracle_mod, state, want)
    for prec, takes, tol in (("fp64", fp64, 1e-12), ("fp32", fp32, 1e-5)):
        s = Solver(c, prec)
        assert rel_l2(s.solve_poisson_equation(rhs)[:n[0], :n[1], :n[2]], phi) <= tol, prec
        s.set_state(*state)
        before = s.launch_count()
        s.compute_time_step_RK3(2)
        assert s.launch_count() - before == 2 * (13 if takes else 19), prec
        got = s.get_state()
        for key, a, b in zip("UVW", got, want):
            assert rel_l2(a, b) <= tol, (prec, key)
        err = rel_l2(interior(c, "P", got[3]), interior(c, "P", want[3]))
        assert err <= p_tol[prec], (prec, "P", err, p_tol[prec])
        s.close()


def test_a_group_and_steps_alone_share_a_context(oracle_mod):
    """A context whose own steps take the one-launch solve, stepped by a group (three launches) and alone in turn."""
    from dfdm.native import Group
    c = cases.channel(64, 64, 64, 3.0, 1.5, 2.0, 2000.0, 1.0, 2e-3, 44, 2, "plane")
    state = cases.initial_condition(c)
    o = oracle_mod.Oracle(c)
    o.set_state(*state)
    o.step(4)
    with Solver(c, "fp32") as s:
        s.set_state(*state)
        s.compute_time_step_RK3(1)
        with Group([s]) as g:
            g.step(1)
            s.compute_time_step_RK3(1)
            s.synchronize()
            g.step(1)
        for key, a, b in zip("UVW", s.get_state(), o.get_state()):
            assert rel_l2(a, b) <= 1e-5, key
