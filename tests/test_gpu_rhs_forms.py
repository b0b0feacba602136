"""The right-hand sides of every form the stage kernels are compiled in (DNS, eddy viscosity, wall model; skew-symmetric and
divergence form, with and without the wall band; periodic and wall-bounded y) on a grid with partial tiles in x and y, and
the wall model on column counts around a block's, against the oracle: FP64 1e-12, FP32 1e-5 relative L2."""
import numpy as np
import pytest

from conftest import interior, rel_l2
from dfdm import cases
from dfdm.native import Solver

pytestmark = pytest.mark.gpu


def _case(wall, sgs, wm, scheme, nwl=-1, nx=62, nz=14, filt=-1):
    if not wall:
        return cases.tgv(16, Re=400.0, name="box").with_(nx=nx, ny=14, nz=nz, sgs_model=sgs, advection_scheme=scheme)
    return cases.Case(name="walls", nx=nx, ny=12, nz=nz, Lx_i=4.0, Ly_i=2.0, Lz_i=1.5, grid_type=2, alpha_grid=2.0, nu=2e-3,
                      dt=1e-3, dPdx=1.0, sgs_model=sgs, flat_wall_model_flag=wm, advection_scheme=scheme,
                      adv_wall_layers=nwl, wm_filter_mode=filt, ic="reichardt_gauss", ic_amplitude=1.0, noise=0.25, seed=5)


def _state(c):
    """The case's mean with noise of a quarter of its amplitude on every component (no component small by symmetry)."""
    U, V, W, P = cases.initial_condition(c)
    rng = np.random.default_rng(9)
    for a in (U, V, W):
        a += rng.normal(0.0, 0.25, size=a.shape)
    cases.fill_ghosts(c, U, V, W)
    return U, V, W, P


FORMS = [(wall, sgs, wm, scheme, nwl) for wall in (True, False) for sgs in (0, 2) for wm in (0, 1) for scheme in (0, 1)
         for nwl in ((-1, 3) if wm else (-1,)) if wall or not wm]


@pytest.mark.parametrize("wall,sgs,wm,scheme,nwl", FORMS)
def test_right_hand_sides(oracle_mod, wall, sgs, wm, scheme, nwl):
    c = _case(wall, sgs, wm, scheme, nwl)
    state = _state(c)
    o = oracle_mod.Oracle(c)
    o.set_state(*state)
    if sgs:
        o.compute_sgs_model()
    if wm:
        o.compute_wall_model(True)
    want = o.compute_rhs()
    Nx, Ny, Nz = c.cells
    rows = (Ny, Ny if c.y_bc_type == 0 else Ny - 1, Ny)
    for prec, variant, tol in (("fp64", None, 1e-12), ("fp32", 0, 1e-5), ("fp32", 1, 1e-5)):
        s = Solver(c, prec)
        if variant is not None:
            s.set_stage_variant(variant)
        s.set_state(*state)
        if sgs:
            s.compute_sgs_model()
        if wm:
            s.compute_wall_model(True)
        for key, n, a, b in zip("uvw", rows, s.compute_rhs(), want):
            assert rel_l2(a[:Nx, :n, :Nz], b[:Nx, :n, :Nz]) <= tol, (prec, variant, key)
        s.close()


@pytest.mark.parametrize("columns", [60, 64, 72, 128])
@pytest.mark.parametrize("filt", [0, 1])
def test_wall_model_columns(oracle_mod, columns, filt):
    c = _case(True, 2, 1, 0, nx=columns + 2, filt=filt)
    state = cases.initial_condition(c)
    o = oracle_mod.Oracle(c)
    o.set_state(*state)
    s = Solver(c, "fp64")
    s.set_state(*state)
    for update in (True, True):
        for a, b in zip(s.compute_wall_model(update), o.compute_wall_model(update)):
            assert rel_l2(a, b) <= 1e-12
    o.step(2)
    s.compute_time_step_RK3(2)
    for key, a, b in zip("UVWP", s.get_state(), o.get_state()):
        assert rel_l2(interior(c, key, a), interior(c, key, b)) <= 1e-12, key
    s.close()
