import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (os.path.join(ROOT, "dopamine-fdm_b200"), os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); parity tests through the C ABI")
    config.addinivalue_line("markers", "slow: long-running case")


def has_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if has_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA GPU in this environment")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


def rel_l2(a, b) -> float:
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    den = np.linalg.norm(b.ravel())
    num = np.linalg.norm((a - b).ravel())
    return float(num / den) if den > 0 else float(num)


def interior(case, key, a):
    """Independent cells of a ghosted reference array (periodic duplicates and ghosts removed)."""
    Nx, Ny, Nz = case.cells
    if key == "V":
        nyv = Ny if case.y_bc_type == 0 else Ny - 1
        return a[1:1 + Nx, 1:1 + nyv, 1:1 + Nz]
    return a[1:1 + Nx, 1:1 + Ny, 1:1 + Nz]


@pytest.fixture(scope="session")
def oracle_mod():
    import oracle as O
    O.build()
    return O


def solve_bound(case):
    """Relative L2 bound of an FP64 pressure solve with y walls: 1e-12, or for many rows the rounding of the pivots of its
    lowest mode, 2^-53 of the largest diagonal entry of d2/dy2 (2/dy_min^2) over the smallest eigenvalue ((pi/Ly)^2)."""
    from dfdm import cases
    y = cases.faces(case)[1]
    return max(1e-12, 2.0 ** -53 * 2.0 / np.diff(y).min() ** 2 / (np.pi / (y[-1] - y[0])) ** 2)


def pressure_bounds(case, oracle_mod, state, want):
    """Relative L2 bounds of P after some steps from `state`, `want` the oracle's state there, for a field whose first
    projection removes much more than the later ones.  P is phi / (0.75 dt) of a weak phi, so what else phi sees counts.
    FP64: the divergence that the first projection leaves, its solve's relative error, enters the next phi whole.
    FP32: the same with eight roundings for the solve, and the rounding of u*: one rounding of the stored velocity (deviations
    from the row means), projected, times sixteen for the operations of the stage update and of the divergence."""
    from dfdm import cases
    n = tuple(case.cells)
    cut = lambda a: np.linalg.norm(a[:n[0], :n[1], :n[2]])

    def phi(U, V, W):
        o = oracle_mod.Oracle(case)
        o.set_state(U, V, W, np.zeros_like(want[3]))
        return cut(o.solve_poisson(o.divergence_rhs()))
    phi2 = 0.75 * case.dt * np.linalg.norm(interior(case, "P", want[3]))
    rng = np.random.default_rng(1)
    noise = []
    for key, a in zip("UVW", want):
        dev = a - a.mean((0, 2), keepdims=True) if key == "U" else a
        noise.append(np.asfortranarray(dev * rng.uniform(-1.0, 1.0, a.shape) * 2.0 ** -24))
    cases.fill_ghosts(case, *noise)
    phi1 = phi(*state[:3])
    return {"fp64": solve_bound(case) * phi1 / phi2, "fp32": (8.0 * 2.0 ** -24 * phi1 + 16.0 * phi(*noise)) / phi2}


def cfl_reference(c, U, V, W, nu_t, dt=None):
    """compute_cfl (src/monitor.f90:304-424) on the ghosted 1-based arrays: i = 2..nxg-1, j = 2..nyg-1,
    k = 2..nzg-1, written out in numpy (0-based slices)."""
    from dfdm import cases
    x, y, z = cases.faces(c)
    dx = np.diff(cases.centres(x)).min()
    idx = 1.0 / dx
    idy = 1.0 / np.maximum(y[1:] - y[:-1], 1e-14)      # index j-2 holds 1/(y(j) - y(j-1)) for j = 2..ny
    idz = 1.0 / np.maximum(z[1:] - z[:-1], 1e-14)
    nxg, nyg, nzg = c.nxg, c.nyg, c.nzg
    I, J, K = slice(1, nxg - 1), slice(1, nyg - 1), slice(1, nzg - 1)
    uc = 0.5 * (U[1:nxg - 1, J, K] + U[0:nxg - 2, J, K])
    vc = 0.5 * (V[I, 1:nyg - 1, K] + V[I, 0:nyg - 2, K])
    wc = 0.5 * (W[I, J, 1:nzg - 1] + W[I, J, 0:nzg - 2])
    iy = idy[0:nyg - 2][None, :, None]
    iz = idz[0:nzg - 2][None, None, :]
    conv = (np.abs(uc) * idx + np.abs(vc) * iy + np.abs(wc) * iz).max()
    visc = ((c.nu + nu_t[I, J, K]) * 2.0 * (idx * idx + iy * iy + iz * iz)).max()
    dt = c.dt if dt is None else dt
    return conv * dt, visc * dt
