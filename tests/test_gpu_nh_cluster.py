"""Small non-hydrostatic grids in one thread-block cluster (nh_clu.cu): the automatic kernel choice
and the brick kernel against the oracle, from one block of a few cells to the largest cluster and
beyond it; the compact cluster kernel where that is the choice; and which kernel is."""
import warnings

import numpy as np
import pytest

from pyom2_b200 import _abi, synth
from pyom2_b200.model import ModelState
from pyom2_b200.non_hydrostatic import NonHydrostatic

pytestmark = pytest.mark.gpu


def tank(nx, ny, nz, cyc_x, cyc_y):
    rng = np.random.default_rng(nx + 31 * ny + 977 * nz)
    M = ModelState(nx, ny, nz, enable_cyclic_x=cyc_x, enable_cyclic_y=cyc_y, coord_degree=False)
    M.dxt[2:nx + 2] = 0.01
    M.dyt[2:ny + 2] = 0.012
    M.dzt[:] = 0.011
    synth.calc_grid(M)
    M.kbot[2:nx + 2, 2:ny + 2] = 1
    M.kbot[2 + nx // 2:4 + nx // 2, 2 + ny // 2] = min(nz, 1 + nz // 2)  # a sill
    M.kbot[2 + nx // 3, 2 + ny // 3] = 0 if ny > 1 else 1  # a column of land
    synth.calc_topo(M)
    forc = np.zeros(M.shape2d + (nz,), order="F")
    inner = (slice(2, -2), slice(2, -2))
    forc[inner] = rng.standard_normal((nx, ny, nz))
    wet = M.maskT > 0
    wet[:2] = wet[-2:] = False
    wet[:, :2] = wet[:, -2:] = False
    forc[wet] -= forc[wet].mean()
    return M, forc


# one block; slices over several blocks, their own neighbours across the seam, odd last pieces; blocks cut in
# y as well, re-entrant both ways; columns of 8 and 12 levels a thread; too deep or too large for the cluster
@pytest.mark.parametrize("nx,ny,nz,cyc_x,cyc_y", [
    (9, 1, 5, False, False), (17, 1, 8, True, False), (64, 1, 24, True, False), (160, 1, 60, True, False),
    (37, 1, 90, False, False), (4, 33, 20, False, True), (24, 17, 7, True, True), (33, 21, 11, False, True),
    (40, 36, 9, False, False), (240, 1, 80, True, False), (48, 40, 24, True, False), (16, 1, 2000, False, False),
    (70, 41, 22, True, True)])
def test_cluster_solve(oracle_lib, nx, ny, nz, cyc_x, cyc_y):
    M, forc = tank(nx, ny, nz, cyc_x, cyc_y)
    O, nh = oracle_lib.Oracle3D(M), NonHydrostatic(M)
    cf = O.make_coeff()
    for it in (1, 4, 12):  # the iterate itself, before rounding has had time to grow
        want = np.zeros(forc.shape, order="F")
        ro = O.congrad(cf, forc, want, eps=0.0, max_it=it)
        for variant in (0, 1):
            nh.set_variant(variant)
            got = np.zeros(forc.shape, order="F")
            with warnings.catch_warnings():
                warnings.simplefilter("ignore")
                n, info = nh.congrad_non_hydro(forc, got, eps=0.0, max_it=it)
            assert n == ro["iterations"] and info["status"] == ro["status"], (variant, it, n, ro)
            assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want), (variant, it)
    nh.close()


# a level's vertical factors are put into shared memory by one warp and read by others: segments of 4, 8 and 12
# levels, columns of more levels than a warp has lanes, one block and several
@pytest.mark.parametrize("nx,ny,nz", [(4, 1, 97), (16, 1, 300), (37, 1, 90), (20, 2, 70), (240, 1, 80), (24, 24, 67),
                                      (96, 4, 100), (60, 60, 12)])
def test_deep_columns_repeat_to_the_bit(oracle_lib, nx, ny, nz):
    M, forc = tank(nx, ny, nz, False, False)
    O, nh = oracle_lib.Oracle3D(M), NonHydrostatic(M)
    want = np.zeros(forc.shape, order="F")
    O.congrad(O.make_coeff(), forc, want, eps=0.0, max_it=5)
    first = None
    for _ in range(20):
        got = np.zeros(forc.shape, order="F")
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            nh.congrad_non_hydro(forc, got, eps=0.0, max_it=5)
        assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)
        first = got if first is None else first
        assert np.array_equal(got, first)
    nh.close()


# 33 600 cells: the cluster kernel's by size, but a brick setting is for the bricks
@pytest.mark.parametrize("call", [("set_grid", 7), ("set_brick", 4, 6), ("set_stages", 3)])
def test_brick_settings_choose_the_bricks(call):
    M, forc = tank(40, 40, 21, True, False)
    out = []
    for variant in (0, 1):
        nh = NonHydrostatic(M)
        nh.set_variant(variant)
        getattr(nh, call[0])(*call[1:])
        p = np.zeros(forc.shape, order="F")
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            nh.congrad_non_hydro(forc, p, eps=0.0, max_it=20)
        out.append(p)
        nh.close()
    assert np.array_equal(*out)


# grids that one cluster of whole columns does not hold: the compact cluster kernel, chosen automatically for deep
# slices and by name up to 110704 cells, with neighbours and halo copies across the seams
@pytest.mark.parametrize("nx,ny,nz,cyc_x,cyc_y,variant", [
    (64, 1, 500, True, False, 0), (5, 5, 1300, True, True, 0), (97, 33, 17, True, False, 2),
    (61, 47, 20, True, True, 2), (40, 60, 30, False, True, 2), (75, 41, 19, False, False, 2)])
def test_compact_cluster_kernel(oracle_lib, nx, ny, nz, cyc_x, cyc_y, variant):
    from torch.profiler import ProfilerActivity, profile
    M, forc = tank(nx, ny, nz, cyc_x, cyc_y)
    O, nh = oracle_lib.Oracle3D(M), NonHydrostatic(M)
    nh.set_variant(variant)
    cf = O.make_coeff()
    start = np.asfortranarray(1e-3 * np.random.default_rng(nx).standard_normal(forc.shape))  # halo unlike the interior
    for it in (1, 4, 12):
        want, got = start.copy(order="F"), start.copy(order="F")
        ro = O.congrad(cf, forc, want, eps=0.0, max_it=it)
        with warnings.catch_warnings(), profile(activities=[ProfilerActivity.CUDA]) as p:
            warnings.simplefilter("ignore")
            n, info = nh.congrad_non_hydro(forc, got, eps=0.0, max_it=it)
        assert any("nh_cg_small_kernel" in e.key for e in p.key_averages())
        assert n == ro["iterations"] and info["status"] == ro["status"], (it, n, ro)
        assert np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want), it
    nh.close()


# one block, several along x, a cut in x and y
CUTS = [(9, 1, 5, False, False), (160, 1, 60, True, False), (24, 17, 7, True, True)]


@pytest.mark.parametrize("nx,ny,nz,cyc_x,cyc_y", CUTS)
def test_timeout_leaves_the_handle_usable(nx, ny, nz, cyc_x, cyc_y):
    M, forc = tank(nx, ny, nz, cyc_x, cyc_y)
    nh = NonHydrostatic(M)
    want, got = (np.zeros(forc.shape, order="F") for _ in range(2))
    n, info = nh.congrad_non_hydro(forc, want, eps=1e-9, max_it=5000)
    assert info["status"] == _abi.OK and n > 3
    nh.set_sync_timeout(0.2)
    nh.inject_barrier_stall(True)
    with pytest.raises(_abi.PyOMGPUError) as e:
        nh.congrad_non_hydro(forc, np.zeros(forc.shape, order="F"), eps=1e-9)
    assert e.value.code == _abi.TIMEOUT
    again, info = nh.congrad_non_hydro(forc, got, eps=1e-9, max_it=5000)
    assert info["status"] == _abi.OK and again == n and np.array_equal(got, want)
    nh.close()


@pytest.mark.parametrize("nx,ny,nz,cyc_x,cyc_y", CUTS)
def test_a_nan_ends_the_solve_and_the_halo_keeps_its_offset(oracle_lib, nx, ny, nz, cyc_x, cyc_y):
    M, forc = tank(nx, ny, nz, cyc_x, cyc_y)
    O, nh = oracle_lib.Oracle3D(M), NonHydrostatic(M)
    start = np.asfortranarray(1e-3 * np.random.default_rng(3).standard_normal(forc.shape))
    want, got = start.copy(order="F"), start.copy(order="F")
    ro = O.congrad(O.make_coeff(), forc, want, eps=0.0, max_it=6)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        n, info = nh.congrad_non_hydro(forc, got, eps=0.0, max_it=6)
    assert n == ro["iterations"] and np.linalg.norm(got - want) <= 1e-10 * np.linalg.norm(want)
    bad = forc.copy(order="F")
    i, j, k = np.argwhere(M.maskT[2:-2, 2:-2] > 0)[5]
    bad[i + 2, j + 2, k] = np.nan
    for variant in (1, 0):
        nh.set_variant(variant)
        with pytest.raises(_abi.PyOMGPUError) as e:
            nh.congrad_non_hydro(bad, np.zeros(forc.shape, order="F"), eps=1e-9)
        assert e.value.code == _abi.NAN, variant
    nh.close()


# deep narrow tanks, whose faces are large for their cells, are slower in the cluster of whole columns; up to 32768
# cells they keep the compact cluster, above it the bricks
@pytest.mark.parametrize("nx,ny,nz,kernel", [
    (160, 1, 60, "nh_clu_kernel"), (8, 8, 100, "nh_clu_kernel"), (60, 60, 12, "nh_clu_kernel"),
    (6, 6, 400, "nh_cg_small_kernel"), (8, 8, 400, "nh_cg_small_kernel"), (16, 16, 170, "nh_cg_kernel"),
    (20, 20, 110, "nh_cg_kernel")])
def test_deep_tanks_keep_the_kernel_that_is_faster(nx, ny, nz, kernel):
    from torch.profiler import ProfilerActivity, profile
    M, forc = tank(nx, ny, nz, False, False)
    nh = NonHydrostatic(M)
    with warnings.catch_warnings(), profile(activities=[ProfilerActivity.CUDA]) as p:
        warnings.simplefilter("ignore")
        nh.congrad_non_hydro(forc, np.zeros(forc.shape, order="F"), eps=0.0, max_it=3)
    assert [k for k in ("nh_clu_kernel", "nh_cg_small_kernel", "nh_cg_kernel")
            if any(k + "<" in e.key for e in p.key_averages())] == [kernel]
    nh.close()
