"""congrad_surf_press (solve_pressure.f90:137-249) on chip: the resident kernel's mask bits,
diagonal term, deferred stop and cyclic halo against the oracle and the tiled kernel."""
import warnings

import numpy as np
import pytest

from pyom2_b200 import synth
from pyom2_b200.external import ExternalMode
from pyom2_b200.model import ModelState

pytestmark = pytest.mark.gpu


def model(nx, ny, cyc_x, cyc_y, seed):
    rng = np.random.default_rng(seed)
    M = ModelState(nx, ny, 1, enable_cyclic_x=cyc_x, enable_cyclic_y=cyc_y, coord_degree=not cyc_y)
    M.dxt[2:nx + 2] = 0.5 if M.coord_degree else 5e4
    M.dyt[2:ny + 2] = min(0.5, 100.0 / ny) if M.coord_degree else 5e4
    M.x_origin, M.y_origin = 0.0, -50.0
    M.dzt[:] = 4000.0
    synth.calc_grid(M)
    M.kbot[2:nx + 2, 2:ny + 2] = synth.smooth_field(rng, (nx, ny), 3.0, (cyc_x, cyc_y)) > -0.05
    M.kbot[3, 3] = 1
    synth.calc_topo(M)
    M.enable_free_surface, M.dt_mom = True, 1800.0
    M.congr_max_iterations = 5000
    forc = np.zeros(M.shape2d, order="F")
    forc[2:-2, 2:-2] = 1e-9 * rng.standard_normal((nx, ny))  # on land too: the solver carries it along
    return M, forc, rng


# the smallest grid, one piece, odd cuts, both cyclic directions, and sizes on each side of the
# points-per-thread instances (4, 8, 16 rows per thread)
@pytest.mark.parametrize("nx,ny,cyc_x,cyc_y", [(4, 4, False, False), (5, 7, True, False), (16, 9, True, True),
                                               (97, 61, True, False), (130, 131, False, False),
                                               (451, 387, True, True), (801, 400, True, False)])
def test_pressure_solve_on_chip(oracle_lib, nx, ny, cyc_x, cyc_y):
    M, forc, rng = model(nx, ny, cyc_x, cyc_y, nx + ny)
    E, O = ExternalMode(M), oracle_lib.Oracle(M)
    start = np.asfortranarray(1e-2 * rng.standard_normal(M.shape2d))  # the halo does not match the interior
    want = start.copy(order="F")
    ro = O.congrad_surf_press(O.make_coeff_surf_press(), forc, want)
    got = {}
    for kernel in ("tiled", "auto"):
        E.set_cg_kernel(kernel)
        p = start.copy(order="F")
        it, info = E.congrad_surf_press(forc, p)
        assert info["status"] == ro["status"] and abs(it - ro["iterations"]) <= 1, (kernel, it, ro)
        got[kernel] = p
    scale = np.linalg.norm(want)
    assert np.linalg.norm(got["auto"] - want) / scale < 1e-10
    assert np.linalg.norm(got["auto"] - got["tiled"]) / scale < 1e-10
    # the iteration limit stops where the oracle stops
    ro = O.congrad_surf_press(O.make_coeff_surf_press(), forc, start.copy(order="F"), max_it=3)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        it, info = E.congrad_surf_press(forc, start.copy(order="F"), max_it=3)
    assert it == ro["iterations"] and info["status"] == ro["status"]
