"""The right-hand sides of every form the stage kernels are compiled in (DNS, eddy viscosity, wall model; skew-symmetric and
divergence form, with and without the wall band; periodic and wall-bounded y) on a grid with partial tiles in x and y, and
the wall model on column counts around a block's, against the oracle: FP64 1e-12, FP32 1e-5 relative L2.  Those fields are
strongly perturbed; the FP32 arithmetic on a smooth mean flow has a test of its own, with a bound in units of its rounding."""
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


@pytest.mark.parametrize("scheme,wm", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_mean_flow_does_not_cancel_in_fp32(oracle_mod, scheme, wm):
    """The u right-hand side of U(y), V(y), W = 0, both exact in FP32, on rows much thinner than the profile changes over:
    -d(uv)/dy is a small difference of large u v at the two faces.  Formed from the differences of u and of v its rounding is
    relative to those: ten roundings at most lie between the stored values and each term (u or its step at the face from two
    weights, three; its partner, two; their product, its metric and the metric's own rounding, three; the sums, two), so the
    error is below 10 x 2^-24 times the sum of the terms' absolute values.  Formed from u v itself it is 4 to 5 times that bound."""
    c = cases.Case(name="mean", nx=34, ny=193, nz=10, Lx_i=6.0, Ly_i=2.0, Lz_i=3.0, grid_type=2, alpha_grid=1.0, nu=1e-4,
                   dt=1e-3, dPdx=1.0, sgs_model=0, flat_wall_model_flag=wm, advection_scheme=scheme,
                   ic="poiseuille_uniform", ic_amplitude=18.0)
    U, V, W, P = cases.initial_condition(c)
    y = cases.faces(c)[1]
    U[:] = U.astype(np.float32)
    V[:] = np.sin(np.pi * y / 2.0).astype(np.float32)[None, :, None]
    V[:, -1] = 0.0
    cases.fill_ghosts(c, U, V, W)
    o = oracle_mod.Oracle(c)
    o.set_state(U, V, W, P)
    if wm:
        o.compute_wall_model(True)
    Nx, Ny, Nz = c.cells
    want = o.compute_rhs()[0][:Nx, 1:Ny - 1, :Nz]          # the wall rows hold the wall model's flux
    g = np.concatenate([[-0.5 * y[1]], 0.5 * (y[1:] + y[:-1]), [2.0 * y[-1] - 0.5 * (y[-1] + y[-2])]])
    u, v = U[1, :, 1], V[1, :, 1]                           # centres with ghosts, faces
    w = (g[1:] - y) / (g[1:] - g[:-1])
    uf, flux = w * u[:-1] + (1.0 - w) * u[1:], c.nu * np.abs(np.diff(u) / np.diff(g))
    big = lambda a: np.maximum(np.abs(a[1:]), np.abs(a[:-1]))
    terms = (np.abs(np.diff(uf)) * big(v) + big(uf) * np.abs(np.diff(v)) + flux[1:] + flux[:-1]) / np.diff(y) + abs(c.dPdx)
    bound = 10.0 * 2.0 ** -24 * np.linalg.norm(np.broadcast_to(terms[None, 1:-1, None], want.shape))
    for variant in (0, 1):
        s = Solver(c, "fp32")
        s.set_stage_variant(variant)
        s.set_state(U, V, W, P)
        if wm:
            s.compute_wall_model(True)
        got = s.compute_rhs()[0][:Nx, 1:Ny - 1, :Nz]
        s.close()
        assert np.linalg.norm(got - want) <= bound, (variant, np.linalg.norm(got - want) / bound)


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
