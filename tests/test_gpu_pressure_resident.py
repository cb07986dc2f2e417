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


# the smallest grid, one piece, odd cuts, both cyclic directions: the automatic choice runs the first five in a
# cluster and the last two on the resident kernel at 8 points a thread
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


# the resident kernel by name (the automatic choice runs the smaller grids in a cluster): 4, 8 and 16 points a
# thread, one row of pieces, odd cuts and both cyclic directions, on grids whose last segments are not whole
@pytest.mark.parametrize("nx,ny,cyc_x,cyc_y,points", [(4, 4, False, False, 4), (16, 9, True, True, 4),
                                                      (97, 61, True, False, 4), (451, 387, True, True, 8),
                                                      (1001, 703, True, True, 16), (1440, 720, True, False, 16)])
def test_pressure_iterates_of_the_resident_kernel(oracle_lib, nx, ny, cyc_x, cyc_y, points):
    M, forc, rng = model(nx, ny, cyc_x, cyc_y, nx + ny)
    E, O = ExternalMode(M), oracle_lib.Oracle(M)
    E.set_cg_kernel("resident")
    assert E.resident_layout()[2] == points
    start = np.asfortranarray(1e-2 * rng.standard_normal(M.shape2d))
    cf = O.make_coeff_surf_press()
    for it in (1, 2, 12):  # the iterate itself, before rounding has had time to grow
        want, got = start.copy(order="F"), start.copy(order="F")
        ro = O.congrad_surf_press(cf, forc, want, max_it=it)
        with warnings.catch_warnings():
            warnings.simplefilter("ignore", RuntimeWarning)
            n, info = E.congrad_surf_press(forc, got, max_it=it)
        assert n == ro["iterations"] and info["status"] == ro["status"], (it, n, ro)
        assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want), it


@pytest.mark.parametrize("nx,ny", [(61, 40), (451, 387)])
def test_a_mask_of_other_values_runs_tiled(oracle_lib, nx, ny):
    M, forc, rng = model(nx, ny, True, False, nx)
    M.maskT[2:-2, 2:-2, -1] *= 0.5 + 0.5 * (rng.random((nx, ny)) < 0.9)  # some cells half wet
    E, O = ExternalMode(M), oracle_lib.Oracle(M)
    want = np.zeros(M.shape2d, order="F")
    ro = O.congrad_surf_press(O.make_coeff_surf_press(), forc, want, max_it=5)
    got = {}
    for kernel in ("auto", "resident", "tiled"):
        E.set_cg_kernel(kernel)
        got[kernel] = np.zeros(M.shape2d, order="F")
        with warnings.catch_warnings():
            warnings.simplefilter("ignore", RuntimeWarning)
            n, info = E.congrad_surf_press(forc, got[kernel], max_it=5)
        assert n == ro["iterations"] and info["status"] == ro["status"]
        assert np.array_equal(got[kernel], got["tiled"] if "tiled" in got else got["auto"])
    assert np.linalg.norm(got["tiled"] - want) <= 1e-10 * np.linalg.norm(want)


@pytest.mark.parametrize("where", ["wet", "land"])
def test_a_nan_ends_the_solve(where):
    from pyom2_b200 import _abi
    M, forc, _ = model(61, 40, True, False, 3)
    wet = M.maskT[2:-2, 2:-2, -1] > 0
    i, j = np.argwhere(wet if where == "wet" else ~wet)[7]
    forc[i + 2, j + 2] = np.nan
    E = ExternalMode(M)
    for kernel in ("tiled", "resident", "auto"):
        E.set_cg_kernel(kernel)
        with pytest.raises(_abi.PyOMGPUError) as e:
            E.congrad_surf_press(forc, np.zeros(M.shape2d, order="F"))
        assert e.value.code == _abi.NAN, kernel
