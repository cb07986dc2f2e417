"""Small grids in one thread-block cluster (cg_clu.cu): the automatic kernel choice against the
oracle and the tiled kernel, on sizes from one block of a few points to the largest cluster."""
import numpy as np
import pytest

from pyom2_b200 import _abi, synth
from pyom2_b200.external import ExternalMode, island_boundaries
from pyom2_b200.model import ModelState

pytestmark = pytest.mark.gpu


def model(nx, ny, cyc_x, cyc_y):
    rng = np.random.default_rng(7 * nx + ny)
    M = ModelState(nx, ny, 1, enable_cyclic_x=cyc_x, enable_cyclic_y=cyc_y, coord_degree=False)
    M.dxt[2:nx + 2] = 2e4
    M.dyt[2:ny + 2] = 2.5e4
    M.dzt[:] = 4000.0
    synth.calc_grid(M)
    M.kbot[2:nx + 2, 2:ny + 2] = 1
    M.kbot[nx // 2 + 1:nx // 2 + 3, ny // 2 + 1:ny // 2 + 3] = 0  # one island
    synth.calc_topo(M)
    depth = 1.0 + 0.5 * rng.random(M.shape2d)
    synth.setcyclic_xy(M, depth)
    for a, r in ((M.hu, M.hur), (M.hv, M.hvr)):
        a *= depth
        r[...] = np.where(a != 0, 1.0 / np.where(a != 0, a, 1.0), 0.0)
    forc = np.zeros(M.shape2d, order="F")
    forc[2:-2, 2:-2] = 1e-12 * rng.standard_normal((nx, ny))
    return M, forc


# one block of 4, 6, 8 points a thread, its own neighbour across a cyclic seam; several blocks with odd
# pieces, both cyclic directions, wide and tall grids; the largest that fit
@pytest.mark.parametrize("nx,ny,cyc_x,cyc_y", [(6, 5, False, False), (7, 9, True, False), (24, 21, False, False),
                                               (33, 23, True, False), (40, 41, False, False), (64, 5, True, True),
                                               (5, 150, False, False), (97, 83, True, False), (211, 101, True, True),
                                               (250, 190, False, False)])
def test_cluster_solve(oracle_lib, nx, ny, cyc_x, cyc_y):
    M, forc = model(nx, ny, cyc_x, cyc_y)
    E, O = ExternalMode(M), oracle_lib.Oracle(M)
    start = np.zeros(M.shape2d, order="F")
    cf = O.make_coeff_streamfunction()
    for it in (1, 7, 40):  # the iterate itself, before rounding has had time to grow
        want, got = start.copy(order="F"), start.copy(order="F")
        ro = O.congrad_streamfunction(cf, forc, want, eps=0.0, max_it=it)
        with pytest.warns(RuntimeWarning) if ro["status"] else _none():
            n, conv, info = E.congrad_streamfunction(forc, got, eps=0.0, max_it=it)
        assert n == ro["iterations"] and info["status"] == ro["status"], (it, n, ro)
        assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)


def _none():
    import contextlib
    return contextlib.nullcontext()


@pytest.mark.parametrize("nx,ny", [(30, 24), (90, 45), (200, 99)])
@pytest.mark.parametrize("precision", [_abi.PREC_F64, _abi.PREC_F32])
def test_cluster_solve_to_residual(nx, ny, precision):
    W = synth.config1(nx=nx, ny=ny)
    E = ExternalMode(W.M)
    b, d, nr = island_boundaries(W.M, maxipp=10**6, maxq=10**6)  # the coasts hold the solution fixed
    W.M.allocate_islands(len(nr), b.shape[1])
    W.M.boundary[...], W.M.line_dir[...], W.M.nr_boundary[...] = b, d, nr
    E.set_islands(with_psin=False)
    out = {}
    for kernel in ("auto", "tiled"):
        E.set_cg_kernel(kernel)
        x = np.zeros(W.M.shape2d, order="F")
        info = E.solve_rtol(W.forc, x, rtol=1e-11, precision=precision)
        assert info["status"] == 0 and info["rel_residual"] <= 1e-11
        out[kernel] = x
    assert np.linalg.norm(out["auto"] - out["tiled"]) <= 1e-8 * np.linalg.norm(out["tiled"])


@pytest.mark.parametrize("nx,ny", [(24, 20), (97, 83), (451, 387)])
def test_the_layout_calls_name_the_kernel_that_runs(nx, ny):
    from torch.profiler import ProfilerActivity, profile
    M, forc = model(nx, ny, False, False)
    E = ExternalMode(M)
    for kernel in ("auto", "resident"):
        E.set_cg_kernel(kernel)
        name, args = E.resident_kernel_name()[:-1].split("<")
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            E.solve_rtol(forc, np.zeros(M.shape2d, order="F"), rtol=1e-3)
        ran = [e.key for e in p.key_averages() if "cg_" in e.key]
        assert len(ran) == 1 and f"{name}<" in ran[0], (name, ran)
        if name == "cg_clu_kernel":
            assert kernel == "auto" and f"<double, {args.replace(',', ', ')}, false>" in ran[0], (args, ran)
        else:
            assert name == "cg_res_kernel" and f"<{args}, " in ran[0], (args, ran)
    npx_npy_nt_p = E.cluster_layout()
    assert (npx_npy_nt_p is None) == (nx * ny > 48000) == (E.cluster_layout(fp32=True) is None)
    if npx_npy_nt_p:
        assert npx_npy_nt_p[0] * npx_npy_nt_p[1] <= 16
