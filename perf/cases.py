"""Performance cases of the library: what an ocean model's program has it do.

Every case is one call (or one model step) through the public Python entry points on arrays that
already live on the GPU, over the sizes of this repository's configurations, tests and benchmark:

===============  =============================================================================
kind             one pass
===============  =============================================================================
``reference``    congrad_streamfunction with the reference's stop (a closed sector: every model
                 step of a coarse set-up makes this call)
``solve``        solve_rtol to an FP64 true relative residual of 2e-11, in FP64 or as FP32 solves
                 with FP64 refinement, on a masked multi-island global grid
``batch``        congrad_streamfunction_batch: closed basins of uneven size in one call
``pressure``     congrad_surf_press: the free-surface variant on the same global grids
``channel``      one hydrostatic model step of the re-entrant channel: momentum tendencies,
                 solve_streamfunction, vertical velocity
``tank``         congrad_non_hydro: the 3-D pressure solve of a non-hydrostatic tank or x-z slice
``learned``      solve_fcg: flexible CG with the learned U-Net preconditioner
``train``        one training step of that network (forward, loss, backward, Adam)
===============  =============================================================================

Grids, masks, depths and forcings are the seeded recipes of ``pyom2_b200.synth`` (smooth-noise land
masks and depths, curl of a smooth forcing), built here without the 3-D mask arrays where the path
does not read them.  ``exact`` computes the same results in 64 bits with plain torch operations:
conjugate gradients in the area-weighted product, in which the operators are self-adjoint, run
to rounding level; explicit expressions for the tendencies; torch's autograd for the network.
"""
import math
import warnings

import numpy as np
import torch
import torch.nn.functional as F

from pyom2_b200 import _abi, learned, synth
from pyom2_b200.external import ExternalMode, congrad_streamfunction_batch, island_boundaries
from pyom2_b200.model import ModelState
from pyom2_b200.non_hydrostatic import NonHydrostatic

NH_EPS = 1e-13  # stop of the 3-D solves on steps of p, whose rms is about 1e-3
RTOL = 2e-11  # residual of the benchmark: solution errors stay below 1e-10 on these operators


# ------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the 2-degree sector of the coarse set-ups: 1600 points, a few hundred iterations, latency only
        {"name": "sector_40x40", "kind": "reference", "nx": 40, "ny": 40},
        # a two-degree global grid with odd sizes, the coarse climate resolution
        {"name": "global_181x91", "kind": "solve", "nx": 181, "ny": 91, "single": False},
        # the quarter-degree global grid, the headline solve
        {"name": "global_1440x720", "kind": "solve", "nx": 1440, "ny": 720, "single": False},
        # the largest grid, with FP32 correction solves inside FP64 refinement
        {"name": "mixed_2048x1024", "kind": "solve", "nx": 2048, "ny": 1024, "single": True},
        # an ensemble of regional basins of uneven size solved in one call
        {"name": "basins_12", "kind": "batch", "count": 12, "smallest": 128, "largest": 512},
        # free-surface set-ups: the pressure solve of a coarse ragged grid and of the quarter-degree grid
        {"name": "pressure_197x99", "kind": "pressure", "nx": 197, "ny": 99, "dt_mom": 3600.0},
        {"name": "pressure_1440x720", "kind": "pressure", "nx": 1440, "ny": 720, "dt_mom": 1800.0},
        # one step of the 0.25-degree ACC channel
        {"name": "channel_256x256x20", "kind": "channel", "nx": 256, "ny": 256, "nz": 20},
        # x-z slice experiments and the 3-D overflow tank of the non-hydrostatic set-ups
        {"name": "slice_160x1x60", "kind": "tank", "nx": 160, "ny": 1, "nz": 60, "cyclic": True},
        {"name": "tank_240x240x80", "kind": "tank", "nx": 240, "ny": 240, "nz": 80, "cyclic": False},
        # the learned preconditioner: a solve with it, and a step of its training
        {"name": "learned_720x360", "kind": "learned", "nx": 720, "ny": 360},
        {"name": "train_1440x720", "kind": "train", "nx": 1440, "ny": 720},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["reference", "solve", "solve", "batch", "pressure", "pressure", "channel", "tank", "tank",
                       "learned", "train"])
    if kind == "reference":
        nx = _log(rng, 24, 160)
        return {"kind": kind, "nx": nx, "ny": max(20, int(nx * rng.uniform(0.6, 1.2)))}
    if kind == "solve":
        single = rng.random() < 0.4
        nx = _log(rng, 240 if single else 96, 2048 if single else 1440)
        return {"kind": kind, "nx": nx, "ny": max(48, nx // 2 - rng.randrange(0, 5)), "single": single}
    if kind == "batch":
        return {"kind": kind, "count": rng.randrange(3, 14), "smallest": _log(rng, 48, 128),
                "largest": _log(rng, 160, 512)}
    if kind == "pressure":
        nx = _log(rng, 96, 1440)
        return {"kind": kind, "nx": nx, "ny": max(48, nx // 2 - rng.randrange(0, 5)),
                "dt_mom": rng.choice([900.0, 1800.0, 3600.0, 7200.0])}
    if kind == "channel":
        nx = _log(rng, 64, 256)
        return {"kind": kind, "nx": nx, "ny": max(48, int(nx * rng.uniform(0.6, 1.0))), "nz": _log(rng, 8, 20)}
    if kind == "tank":
        if rng.random() < 0.4:
            return {"kind": kind, "nx": _log(rng, 64, 256), "ny": 1, "nz": _log(rng, 20, 80),
                    "cyclic": rng.random() < 0.5}
        nx = _log(rng, 40, 240)
        return {"kind": kind, "nx": nx, "ny": max(8, int(nx * rng.uniform(0.5, 1.0))), "nz": _log(rng, 10, 80),
                "cyclic": rng.random() < 0.5}
    nx = _log(rng, 192, 720 if kind == "learned" else 1440)
    return {"kind": kind, "nx": nx, "ny": max(96, nx // 2 - rng.randrange(0, 9))}


# ------------------------------------------------------------------------------------- inputs
def _dev(a):
    """Fortran-ordered CUDA tensor of a host array."""
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().permute(*reversed(range(np.ndim(a))))


def _zeros(shape):
    return torch.zeros(tuple(reversed(shape)), dtype=torch.float64, device="cuda").permute(
        *reversed(range(len(shape))))


def _depths(M, H):
    """Column depths at the u and v points from the interior T-cell depth H."""
    X, Y = M.shape2d
    h = np.zeros((X, Y), order="F")
    h[2:-2, 2:-2] = H
    synth.setcyclic_xy(M, h)
    M.hu[...] = 0.0
    M.hv[...] = 0.0
    M.hu[:-1] = np.minimum(h[:-1], h[1:]) * M.maskU[:-1, :, -1]
    M.hv[:, :-1] = np.minimum(h[:, :-1], h[:, 1:]) * M.maskV[:, :-1, -1]
    synth.setcyclic_xy(M, M.hu)
    synth.setcyclic_xy(M, M.hv)
    for r, d in ((M.hur, M.hu), (M.hvr, M.hv)):
        r[...] = np.where(d != 0.0, 1.0 / np.where(d != 0.0, d, 1.0), 0.0)


def _globe(nx, ny, seed):
    """Cyclic 80S-80N grid, ~30 % land in at most 20 masses, 500-5500 m deep (one level stored)."""
    rng = np.random.default_rng(np.random.PCG64(seed))
    M = ModelState(nx, ny, 1, enable_cyclic_x=True, coord_degree=True)
    M.dxt[2:nx + 2] = 360.0 / nx
    M.dyt[2:ny + 2] = 160.0 / ny
    M.x_origin, M.y_origin = 0.0, -80.0
    M.dzt[:] = 5500.0
    synth.calc_grid(M)
    noise = synth.smooth_field(rng, (nx, ny), max(2.0, nx / 72.0), (True, False))
    land = synth.clean_land_mask(noise < np.quantile(noise, 0.30), cyclic_x=True, keep_islands=18)
    M.kbot[2:nx + 2, 2:ny + 2] = np.where(land, 0, 1)
    synth.calc_topo(M)
    d = synth.smooth_field(rng, (nx, ny), max(2.0, nx / 60.0), (True, False))
    _depths(M, np.where(land, 0.0, 500.0 + 5000.0 * (d - d.min()) / (d.max() - d.min())))
    return M, rng


def _basin(nx, ny, rng):
    """Closed quarter-degree basin from 60S, 10-40 % land, up to 12 interior islands."""
    M = ModelState(nx, ny, 1, enable_cyclic_x=False, coord_degree=True)
    M.dxt[2:nx + 2] = 0.25
    M.dyt[2:ny + 2] = min(0.25, 100.0 / ny)
    M.x_origin, M.y_origin = 0.0, -60.0
    M.dzt[:] = 5500.0
    synth.calc_grid(M)
    noise = synth.smooth_field(rng, (nx, ny), max(4.0, max(nx, ny) / 40.0), (False, False))
    land = synth.clean_land_mask(noise < np.quantile(noise, float(rng.uniform(0.1, 0.4))), cyclic_x=False,
                                 keep_islands=int(rng.integers(0, 13)))
    M.kbot[2:nx + 2, 2:ny + 2] = np.where(land, 0, 1)
    synth.calc_topo(M)
    d = synth.smooth_field(rng, (nx, ny), max(nx, ny) / 50.0, (False, False))
    _depths(M, np.where(land, 0.0, 500.0 + 5000.0 * (d - d.min()) / (d.max() - d.min())))
    return M


def _islands(M):
    """Island perimeters (the reference's lists) on M; psin is not needed by the solves."""
    b, d, nr = island_boundaries(M, maxipp=10**6, maxq=10**6)
    M.allocate_islands(len(nr), b.shape[1])
    M.boundary[...], M.line_dir[...], M.nr_boundary[...] = b, d, nr
    E = ExternalMode(M)
    E.set_islands(M, with_psin=False)
    return E


def _forcing(M, rng, sigma=5.0):
    fpx, fpy = synth.random_fp(M, rng, sigma=sigma, rms=1e-7)
    return synth.forcing_from_fp(M, fpx, fpy)


def _channel(case, seed):
    """The re-entrant channel with a velocity, density and streamfunction history: smooth eddies of
    0.1 m/s, 0.1 K of temperature noise on a linear stratification, and a slowly changing dpsi."""
    from pyom2_b200.sequence import RHO_NOISE, channel_physics
    W = synth.config4(seed, nx=case["nx"], ny=case["ny"], nz=case["nz"])
    M = W.M
    channel_physics(M)
    rng = np.random.default_rng(np.random.PCG64(seed + 17))
    shape3, cyc = M.shape2d + (M.nz,), (True, False, False)

    def field(mask, rms, sig=(8.0, 8.0, 2.0)):
        f = synth.smooth_field(rng, shape3, sig, cyc)
        f = np.asfortranarray(f * (rms / math.sqrt(np.mean(f * f))) * mask)
        synth.setcyclic_xy(M, f)
        return f

    u, v, w = field(M.maskU, 0.1), field(M.maskV, 0.1), field(M.maskW, 1e-5)
    rho = np.asfortranarray(M.maskT * (1024.0 - 2.0 * M.zt / 4000.0)[None, None, :] + field(M.maskT, RHO_NOISE))
    for lev in range(3):
        M.u[..., lev], M.v[..., lev], M.w[..., lev], M.rho[..., lev] = u, v, w, rho
        M.du[..., lev] = field(M.maskU, 1e-7) if lev == 0 else 0.0
        M.dv[..., lev] = field(M.maskV, 1e-7) if lev == 0 else 0.0
    s = synth.smooth_field(rng, M.shape2d, 12.0, (True, False))
    s *= 10.0 / math.sqrt(np.mean(s * s))
    E = ExternalMode(M)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        E.streamfunction_init(maxipp=10**6, maxq=10**6, psin_rtol=1e-13, psin_weighted=True)
    s[2:-2, 2:-2] *= _operator(M)["unk"].cpu().numpy().T  # zero on the coasts, as the model keeps it
    s[:, :2] = s[:, -2:] = 0.0
    synth.setcyclic_xy(M, s)
    M.dpsi[..., 0], M.dpsi[..., 1] = 0.99 * s, s
    M.psi[..., 1] = 1e5 * s
    M.dpsin[:, 0] = 100.0 * rng.standard_normal(M.nisle)
    host = {n: np.array(getattr(M, n), order="F") for n in ("u", "v", "w", "du", "dv", "rho", "dpsi", "psi", "psin",
                                                            "dpsin", "line_psin")}
    for n in ("u", "v", "w", "du", "dv", "rho", "du_mix", "dv_mix", "p_hydro", "psi", "dpsi", "dpsin", "dzt", "dzw",
              "tantr", "maskT", "maskU", "maskV", "maskW", "coriolis_t", "area_t", "area_u", "area_v",
              "surface_taux", "surface_tauy", "kappaM"):
        setattr(M, n, _dev(getattr(M, n)))
    # the model's arrays stay on the GPU; kbot as momentum passes it on
    M.kbot = torch.from_numpy(np.ascontiguousarray(np.asarray(M.kbot, dtype=np.int32).T)).cuda()
    return {"M": M, "E": E, "host": host}


def _tank(case, seed):
    """Tank of synth.nonhydro_tank: shelf and rough slope, divergence of a smooth velocity field."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    W = synth.nonhydro_tank(nx, ny, nz, seed, cyclic_x=case["cyclic"])
    return W.M, W.forc


def _pair(M, seed):
    """A training pair (r, e): the error is a smooth random field on the unknowns, r = A e."""
    rng = np.random.default_rng(np.random.PCG64(seed + 5))
    op = _operator(M)
    e = np.zeros(M.shape2d, order="F")
    e[2:-2, 2:-2] = synth.smooth_field(rng, (M.nx, M.ny), 6.0, (True, False)) * op["unk"].cpu().numpy().T
    r = np.zeros(M.shape2d, order="F")
    r[2:-2, 2:-2] = (_apply(op, torch.from_numpy(np.ascontiguousarray(e[2:-2, 2:-2].T)).cuda())
                     * op["unk"]).cpu().numpy().T
    for a in (e, r):
        synth.setcyclic_xy(M, a)
    return _dev(r), _dev(e)


def prepare(case, seed):
    return dict(_inputs(case, seed), case=case)


def _inputs(case, seed):
    kind = case["kind"]
    if kind == "reference":
        M, forc = _sector(case, seed)
        return {"E": _islands(M), "M": M, "forc": _dev(forc), "sol": _zeros(M.shape2d)}
    if kind in ("solve", "pressure", "learned", "train"):
        M, rng = _globe(case["nx"], case["ny"], seed)
        if kind == "pressure":
            M.enable_free_surface = True
            M.dt_mom = case["dt_mom"]
            M.congr_max_iterations = 100000
            E, forc = ExternalMode(M), _press_forcing(M, rng)
        else:
            E, forc = _islands(M), None if kind == "train" else _forcing(M, rng)
        S = {"E": E, "M": M}
        if kind == "train":
            S["r"], S["e"] = _pair(M, seed)
            S["net"] = learned.LearnedPreconditioner(E, params=learned.init_params(seed), training=True)
            return S
        if kind == "learned":
            S["net"] = learned.LearnedPreconditioner(E, params=learned.load_params())
        return dict(S, forc=_dev(forc), sol=_zeros(M.shape2d))
    if kind == "batch":
        Ms, forcs = _basins(case, seed)
        return {"E": [_islands(M) for M in Ms], "M": Ms, "forc": [_dev(f) for f in forcs],
                "sol": [_zeros(M.shape2d) for M in Ms]}
    if kind == "channel":
        return _channel(case, seed)
    M, forc = _tank(case, seed)
    return {"E": NonHydrostatic(M), "M": M, "forc": _dev(forc), "sol": _zeros(M.shape2d + (M.nz,))}


def _sector(case, seed):
    """The closed two-degree sector of synth.config0 at the case's size: land ring, one island, ridge."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng(np.random.PCG64(seed))
    M = ModelState(nx, ny, 1, enable_cyclic_x=False, coord_degree=True)
    M.dxt[2:nx + 2] = 80.0 / nx
    M.dyt[2:ny + 2] = 80.0 / ny
    M.x_origin, M.y_origin = 0.0, -40.0
    M.dzt[:] = 4000.0
    synth.calc_grid(M)
    wet = np.ones((nx, ny), dtype=bool)
    wet[0] = wet[-1] = wet[:, 0] = wet[:, -1] = False
    wet[nx // 2 - 2:nx // 2 + 2, ny // 2 - 2:ny // 2 + 2] = False
    M.kbot[2:nx + 2, 2:ny + 2] = wet
    synth.calc_topo(M)
    i = np.arange(nx)[:, None]
    _depths(M, np.where(wet, 4000.0 - 1500.0 * np.exp(-(i - nx * rng.uniform(0.4, 0.6)) ** 2 / (2 * 8.0 ** 2)), 0.0))
    M.congr_max_iterations = 20000
    return M, _forcing(M, rng)


def _basins(case, seed):
    sizes = np.random.default_rng(case["count"])  # the sizes are the case's; masks, depths and forcings the seed's
    rng = np.random.default_rng(np.random.PCG64(seed))
    Ms, forcs = [], []
    for _ in range(case["count"]):
        n = sizes.integers(case["smallest"], case["largest"] + 1, 2)
        Ms.append(_basin(int(n[0]), max(32, int(0.75 * n[1])), rng))
        forcs.append(_forcing(Ms[-1], rng))
    return Ms, forcs


def _press_forcing(M, rng):
    """Divergence forcing of solve_pressure: smooth transport divergences over dt on the wet cells."""
    f = np.zeros(M.shape2d, order="F")
    g = synth.smooth_field(rng, (M.nx, M.ny), 4.0, (True, False))
    f[2:-2, 2:-2] = 1e-9 * g / math.sqrt(np.mean(g * g)) * M.maskT[2:-2, 2:-2, -1]
    return f


# ------------------------------------------------------------------------------------- one pass
def run(S):
    M, E, kind = S["M"], S["E"], S["case"]["kind"]
    if kind == "channel":
        E.momentum(M)
        E.solve_streamfunction(M)
        E.vertical_velocity(M)
        t0, t1 = M.tau - 1, M.taup1 - 1
        return {"u": M.u[..., t1], "v": M.v[..., t1], "w": M.w[..., t1], "psi": M.psi[..., t1],
                "dpsi": M.dpsi[..., t1], "du": M.du[..., t0], "dv": M.dv[..., t0], "du_mix": M.du_mix,
                "dv_mix": M.dv_mix, "p_hydro": M.p_hydro, "dpsin": M.dpsin[:, t0]}
    if kind == "train":
        # a small learning rate, as late in training; the step computes its loss in 32 bits
        loss = S["net"].train_step(S["r"], S["e"], 1e-6)
        return {"loss": np.float32(loss), "grads": S["net"].get_grads()}
    for x in S["sol"] if kind == "batch" else [S["sol"]]:
        x.zero_()
    if kind == "batch":
        congrad_streamfunction_batch(E, S["forc"], S["sol"], eps=0.0, rtol=RTOL)
    elif kind == "tank":
        E.congrad_non_hydro(S["forc"], S["sol"], eps=NH_EPS, max_it=20000)
    elif kind == "learned":
        learned.solve_fcg(E, S["net"], S["forc"], S["sol"], rtol=RTOL)
    elif kind == "pressure":
        E.congrad_surf_press(S["forc"], S["sol"])
    elif kind == "solve":
        E.solve_rtol(S["forc"], S["sol"], rtol=RTOL,
                     precision=_abi.PREC_F32 if S["case"]["single"] else _abi.PREC_F64)
    else:
        E.congrad_streamfunction(S["forc"], S["sol"])
    return S["sol"]


def work(case):
    """Bytes: every input field read once and every output written once.  Operations of the iterative
    solves: about 20 per point and iteration of Jacobi-preconditioned CG, whose iteration count on these
    grids is about 1.3 times the longer side (a tenth of it with the mass term of the free surface)."""
    kind = case["kind"]
    if kind == "batch":
        n = (0.5 * (case["smallest"] + case["largest"])) ** 2 * 0.75 * case["count"]
        return {"bytes": n * 8 * 5, "flops": n * 20 * 1.3 * case["largest"]}
    n = case["nx"] * case["ny"]
    long = max(case["nx"], case["ny"])
    if kind == "tank":
        n *= case["nz"]
        return {"bytes": n * 17, "flops": n * 25 * 5 * max(long, case["nz"])}
    if kind == "channel":
        c = n * case["nz"]
        # u, v, w, rho, du, dv history, masks, viscosity in; u, v, w, du, dv, du_mix, dv_mix, p_hydro out
        return {"bytes": 8 * (c * (10 + 8) + n * 20), "flops": c * 300 + n * 20 * 4 * long}
    if kind in ("learned", "train"):
        macs = sum(ci * co * 9 / 4 ** lev for (ci, co), lev in
                   zip(learned.LAYERS, (0, 0, 1, 1, 2, 2, 3, 3, 3, 2, 1, 0)))
        if kind == "train":
            return {"bytes": n * (8 * 2 + 2 * 2 * 16 * 4), "flops": 6 * macs * n}
        return {"bytes": n * 8 * 5, "flops": n * (2 * macs + 100) * 0.65 * long}
    per = 0.13 if kind == "pressure" else 1.3
    return {"bytes": n * 8 * 5, "flops": n * 20 * per * long}


# ------------------------------------------------------------------------------------- 64 bits
def _t(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, dtype=np.float64).T)).cuda()


def _operator(M, pressure=False):
    """The five-point operator A = D^-1 S on the interior (tensors (ny, nx)): couplings across the
    west/east and south/north faces of S, cell weight D, diagonal of S and the unknowns."""
    nx, ny = M.nx, M.ny
    I, J = slice(2, nx + 2), slice(2, ny + 2)
    dxt, dxu, dyt, dyu, cost, cosu = (_t(getattr(M, n)) for n in ("dxt", "dxu", "dyt", "dyu", "cost", "cosu"))
    if pressure:  # make_coeff_surf_press, solve_pressure.f90:87-131
        hu, hv, m = _t(M.hu), _t(M.hv), _t(M.maskT[:, :, -1])
        D = (cost[J] * dyt[J])[:, None] * dxt[I][None, :]
        fx = m[:, 1:] * m[:, :-1] * hu[:, :-1] / dxu[None, :-1]                    # face west of column i, from i = 1
        fy = m[1:] * m[:-1] * hv[:-1] * (cosu / dyu)[:-1, None]
        cw = (dyt / cost)[J][:, None] * fx[J, 1:nx + 1]
        ce = (dyt / cost)[J][:, None] * fx[J, 2:nx + 2]
        cs, cn = dxt[I][None, :] * fy[1:ny + 1, I], dxt[I][None, :] * fy[2:ny + 2, I]
        mass = m[J, I] / (M.grav * M.dt_mom ** 2) * D
        unk = m[J, I] != 0
    else:  # make_coeff_streamfunction, solve_streamfct.f90:123-148
        hur, hvr = _t(M.hur), _t(M.hvr)
        D = (cosu[J] * dyu[J])[:, None] * dxu[I][None, :]
        fx, fy = hvr / dxt[None, :], hur * (cost / dyt)[:, None]
        cw = (dyu / cosu)[J][:, None] * fx[J, I]
        ce = (dyu / cosu)[J][:, None] * fx[J, 3:nx + 3]
        cs, cn = dxu[I][None, :] * fy[J, I], dxu[I][None, :] * fy[3:ny + 3, I]
        mass = torch.zeros_like(D)
        unk = (cw + ce + cs + cn) != 0
        per = np.zeros(M.shape2d, dtype=bool)
        for k in range(M.nisle):
            b = M.boundary[k, :M.nr_boundary[k]]
            per[b[:, 0] + 1, b[:, 1] + 1] = True
        unk &= ~torch.from_numpy(np.ascontiguousarray(per[2:-2, 2:-2].T)).cuda()
    return {"cw": cw, "ce": ce, "cs": cs, "cn": cn, "D": D, "mass": mass, "unk": unk, "cyclic": M.enable_cyclic_x}


def _apply(op, p, south=None, north=None):
    """A p on the interior; p is zero outside a closed side."""
    q = F.pad(p[None, None], (1, 1, 0, 0), mode="circular" if op["cyclic"] else "constant")
    q = F.pad(q, (0, 0, 1, 1))[0, 0]
    s = (op["ce"] * (q[1:-1, 2:] - p) + op["cw"] * (q[1:-1, :-2] - p) + op["cn"] * (q[2:, 1:-1] - p)
         + op["cs"] * (q[:-2, 1:-1] - p) - op["mass"] * p)
    return s / op["D"]


def _solve(apply, D, diag, unk, f, x, passes=3, tol=1e-14, most=60000):
    """D A x = D f on the unknowns by Jacobi-preconditioned conjugate gradients in the D product, restarted
    from the true residual `passes` times; the other points keep their value."""
    unk = unk.to(torch.float64)
    inv = torch.where(unk > 0, 1.0 / torch.where(diag != 0, diag, torch.ones_like(diag)), torch.zeros_like(diag))
    ref = None
    for _ in range(passes):
        r = (f - apply(x)) * D * unk
        z = inv * r
        rz = torch.sum(r * z)
        ref = rz.abs() if ref is None else ref
        p = z.clone()
        for it in range(most):
            q = apply(p) * D * unk
            a = rz / torch.sum(p * q)
            x = x + a * p
            r = r - a * q
            z = inv * r
            new = torch.sum(r * z)
            p = z + (new / rz) * p
            rz = new
            if it % 50 == 49 and float((rz / ref).abs()) < tol * tol:
                break
    return x


def _solve2(M, f, x, pressure=False):
    op = _operator(M, pressure)
    diag = -(op["cw"] + op["ce"] + op["cs"] + op["cn"] + op["mass"])
    return _solve(lambda p: _apply(op, p), op["D"], diag, op["unk"], f, x)


def _whole(M, x, halo):
    """(nx+4, ny+4) of an interior solution from a zero guess, with the cyclic halo where the call fills it."""
    out = F.pad(x, (2, 2, 2, 2))
    if halo and M.enable_cyclic_x:
        out[:, :2], out[:, -2:] = out[:, -4:-2].clone(), out[:, 2:4].clone()
    return out.T


def _inner(a):
    return _t(a)[..., 2:-2, 2:-2]


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_whole(M, _solve2(M, _inner(f), torch.zeros_like(_inner(f))), True)
                for M, f in zip(*_with_islands(*_basins(case, seed)))]
    if kind == "tank":
        return _exact_tank(*_tank(case, seed))
    if kind == "channel":
        return _exact_channel(_channel(case, seed))
    S = prepare(case, seed)
    M = S["M"]
    if kind == "train":
        return _exact_train(S)
    f = S["forc"].T[2:-2, 2:-2].contiguous()
    return _whole(M, _solve2(M, f, torch.zeros_like(f), kind == "pressure"), kind != "reference")


def _with_islands(Ms, forcs):
    for M in Ms:
        _islands(M)
    return Ms, forcs


def _exact_tank(M, forc):
    """The seven-point operator of make_coeff_non_hydro (non_hydrostatic.f90:70-138) on (nz, ny, nx); with
    equal cells the solution from a zero guess has zero mean over the wet cells."""
    nx, ny, nz = M.nx, M.ny, M.nz
    mU, mV, mW, mT = (_t(getattr(M, n)) for n in ("maskU", "maskV", "maskW", "maskT"))
    J, I = slice(2, ny + 2), slice(2, nx + 2)
    dx, dz = float(M.dxt[2]), float(M.dzt[0])
    top = mW[:, J, I].clone()
    top[-1] = 0.0
    ce, cw, cn, cs = mU[:, J, I], mU[:, J, 1:nx + 1], mV[:, J, I], mV[:, 1:ny + 1, I]
    cs, cn = cs / dx ** 2, cn / dx ** 2
    ce, cw, ct = ce / dx ** 2, cw / dx ** 2, top / dz ** 2
    cb = torch.zeros_like(ct)
    cb[1:] = ct[:-1]
    diag = -(ce + cw + cn + cs + ct + cb)
    pad = "circular" if M.enable_cyclic_x else "constant"

    def apply(p):
        q = F.pad(p[None], (1, 1, 0, 0), mode=pad)[0]
        a = diag * p + ce * q[..., 2:] + cw * q[..., :-2]
        a[:, :-1] += cn[:, :-1] * p[:, 1:]
        a[:, 1:] += cs[:, 1:] * p[:, :-1]
        a[:-1] += ct[:-1] * p[1:]
        a[1:] += cb[1:] * p[:-1]
        return a

    wet = mT[:, J, I]
    f = _t(forc)[:, J, I]
    x = _solve(apply, torch.ones_like(f), diag, (wet > 0) & (diag != 0), f, torch.zeros_like(f))
    x = (x - (x * wet).sum() / wet.sum()) * wet
    out = F.pad(x, (2, 2, 2, 2))
    if M.enable_cyclic_x:
        out[..., :2], out[..., -2:] = out[..., -4:-2].clone(), out[..., 2:4].clone()
    return out.permute(2, 1, 0)


def _exact_channel(S):
    """momentum.f90:4-152, solve_streamfct.f90:10-120 and vertical_velocity.f90 on (nz, ny+4, nx+4)."""
    M, host = S["M"], S["host"]
    nx, ny, nz = M.nx, M.ny, M.nz
    dxt, dxu, dyt, dyu, cost, cosu = (_t(getattr(M, n)) for n in ("dxt", "dxu", "dyt", "dyu", "cost", "cosu"))
    g = {n: getattr(M, n).permute(*reversed(range(getattr(M, n).dim()))) for n in (
        "maskT", "maskU", "maskV", "maskW", "coriolis_t", "area_t", "area_u", "area_v", "surface_taux",
        "surface_tauy", "kappaM", "dzt", "dzw", "tantr")}
    mT, mU, mV, mW, cor = g["maskT"], g["maskU"], g["maskV"], g["maskW"], g["coriolis_t"]
    dzt, dzw = g["dzt"][:, None, None], g["dzw"][:, None, None]
    u, v, w = (_t(host[n][..., 1]) for n in ("u", "v", "w"))
    rho = _t(host["rho"][..., 1])
    kb = M.kbot

    def X(a):  # a 1-D factor in x / y as a field
        return a[None, :]

    def Y(a):
        return a[:, None]

    def s(a, di=0, dj=0):  # a(i+di, j+dj) on the interior
        return a[..., 2 + dj:ny + 2 + dj, 2 + di:nx + 2 + di]

    def full(a):
        return F.pad(a, (2, 2, 2, 2))

    dxt2, dxu2, dyt2, dyu2 = (q.expand(ny + 4, nx + 4) for q in (X(dxt), X(dxu), Y(dyt), Y(dyu)))
    ct2, cu2, tan2 = (Y(q).expand(ny + 4, nx + 4) for q in (cost, cosu, g["tantr"]))
    # Coriolis and metric terms
    vb = v + F.pad(v, (0, 0, 1, 0))[:, :-1]                    # v(i,j) + v(i,j-1)
    ub = u + F.pad(u, (1, 0))[..., :-1]                        # u(i-1,j) + u(i,j)
    du = s(mU) * 0.25 * (s(cor) * s(vb) * s(dxt2) + s(cor, 1) * s(vb, 1) * s(dxt2, 1)) / s(dxu2)
    dv = -s(mV) * 0.25 * (s(cor) * s(ub) * s(dyt2) * s(ct2) + s(cor, 0, 1) * s(ub, 0, 1) * s(dyt2, 0, 1)
                          * s(ct2, 0, 1)) / (s(dyu2) * s(cu2))
    du = du + s(mU) * 0.125 * s(tan2) * (s(ub) * s(vb) * s(dxt2) + s(ub, 1) * s(vb, 1) * s(dxt2, 1)) / s(dxu2)
    dv = dv - s(mV) * 0.125 * (s(tan2) * s(ub) ** 2 * s(dyt2) * s(ct2) + s(tan2, 0, 1) * s(ub, 0, 1) ** 2
                               * s(dyt2, 0, 1) * s(ct2, 0, 1)) / (s(dyu2) * s(cu2))
    du[-1] += s(mU)[-1] * s(g["surface_taux"]) / dzt[-1]
    dv[-1] += s(mV)[-1] * s(g["surface_tauy"]) / dzt[-1]
    # advection
    ut, vt, wt = dzt * dyt2 * u * mU, dzt * cu2 * dxt2 * v * mV, g["area_t"] * w * mW
    for q, mask, area, out, e in ((u, mU, g["area_u"], du, (1, 0)), (v, mV, g["area_v"], dv, (0, 1))):
        fe = 0.25 * (s(q) + s(q, 1)) * (s(ut) + s(ut, *e))
        fw = 0.25 * (s(q) + s(q, -1)) * (s(ut, -1) + s(ut, e[0] - 1, e[1]))
        fn = 0.25 * (s(q) + s(q, 0, 1)) * (s(vt) + s(vt, *e))
        fs = 0.25 * (s(q) + s(q, 0, -1)) * (s(vt, 0, -1) + s(vt, e[0], e[1] - 1))
        ft = torch.zeros_like(fe)
        ft[:-1] = 0.25 * (s(q)[1:] + s(q)[:-1]) * (s(wt) + s(wt, *e))[:-1]
        fb = torch.zeros_like(fe)
        fb[1:] = ft[:-1]
        out -= s(mask) * (fe - fw + fn - fs + ft - fb) / (s(area) * dzt)
    # implicit vertical friction, harmonic and bottom friction
    mix = []
    for q, mask, e in ((u, mU, (1, 0)), (v, mV, (0, 1))):
        m = s(mask)
        ks = torch.maximum(s(kb), s(kb, *e)).long()
        lev = torch.arange(1, nz + 1, device="cuda")[:, None, None]
        inside = (ks > 0) & (lev >= ks)
        d = torch.zeros_like(m)
        d[:-1] = (M.dt_mom / dzw * 0.5 * (s(g["kappaM"]) + s(g["kappaM"], *e)) * m)[:-1] * m[1:]
        d[:-1] = torch.where(inside[:-1], d[:-1], torch.zeros_like(d[:-1]))
        low = torch.zeros_like(d)
        low[1:] = d[:-1]
        a, c = -low / dzt, -d / dzt
        b = 1 - a - c
        cp, dp = torch.zeros_like(d), torch.zeros_like(d)
        for k in range(nz):
            den = b[k] - (cp[k - 1] * a[k] if k else 0.0)
            cp[k] = c[k] / den
            dp[k] = (s(q)[k] - (dp[k - 1] * a[k] if k else 0.0)) / den
        x = torch.zeros_like(d)
        x[-1] = dp[-1]
        for k in range(nz - 2, -1, -1):
            x[k] = dp[k] - cp[k] * x[k + 1]
        mx = torch.where(inside, (x - s(q)) / M.dt_mom, torch.zeros_like(x))
        # flux_east and flux_north of harmonic_friction.f90 (cos scaling), at (i, j) and its west / south faces
        if e == (1, 0):
            fe = lambda di: s(ct2) * M.A_h * (s(q, di + 1) - s(q, di)) / (s(ct2) * s(dxt2, di + 1)) * s(mask, di + 1) * s(mask, di)
            fn = lambda dj: s(cu2, 0, dj) * M.A_h * (s(q, 0, dj + 1) - s(q, 0, dj)) / s(dyu2, 0, dj) * s(mask, 0, dj + 1) * s(mask, 0, dj) * s(cu2, 0, dj)
            mx = mx + m * ((fe(0) - fe(-1)) / (s(ct2) * s(dxu2)) + (fn(0) - fn(-1)) / (s(ct2) * s(dyt2)))
        else:
            fe = lambda di: s(cu2) * M.A_h * (s(q, di + 1) - s(q, di)) / (s(cu2) * s(dxu2, di)) * s(mask, di + 1) * s(mask, di)
            fn = lambda dj: s(ct2, 0, dj + 1) * M.A_h * (s(q, 0, dj + 1) - s(q, 0, dj)) / s(dyt2, 0, dj + 1) * s(ct2, 0, dj + 1) * s(mask, 0, dj) * s(mask, 0, dj + 1)
            mx = mx + m * ((fe(0) - fe(-1)) / (s(cu2) * s(dxt2)) + (fn(0) - fn(-1)) / (s(cu2) * s(dyu2)))
        mx = mx - torch.where(lev == ks, m * M.r_bot * s(q), torch.zeros_like(mx))
        mix.append(full(mx))
    du_mix, dv_mix = mix
    # hydrostatic pressure and its gradient
    ph = torch.zeros_like(rho)
    fxa = M.grav / M.rho_0
    ph[-1] = 0.5 * rho[-1] * fxa * dzw[-1] * mT[-1]
    for k in range(nz - 2, -1, -1):
        ph[k] = mT[k] * (ph[k + 1] + 0.5 * (rho[k + 1] + rho[k]) * fxa * dzw[k])
    du = full(du - (s(ph, 1) - s(ph)) / (s(dxu2) * s(ct2)) * s(mU))
    dv = full(dv - (s(ph, 0, 1) - s(ph)) / s(dyu2) * s(mV))
    hur, hvr = _t(M.hur), _t(M.hvr)
    fpx = ((du + du_mix) * mU * dzt).sum(0) * hur
    fpy = ((dv + dv_mix) * mV * dzt).sum(0) * hvr
    for q in (fpx, fpy):
        q[:, :2], q[:, -2:] = q[:, -4:-2].clone(), q[:, 2:4].clone()
    forc = (s(fpy, 1) - s(fpy)) / (s(cu2) * s(dxu2)) - (s(ct2, 0, 1) * s(fpx, 0, 1) - s(ct2) * s(fpx)) / (
        s(cu2) * s(dyu2))
    dp0, dpm = _t(host["dpsi"][..., 1]), _t(host["dpsi"][..., 0])
    dp1 = _whole(M, _solve2(M, forc, s(2 * dp0 - dpm)), True).T.contiguous()
    # island line integrals (streamfct_init.f90:311-377) and the island system
    psi = dp1
    up, vp = torch.zeros_like(psi), torch.zeros_like(psi)
    up[1:] = -(mU[-1] * hur / dyt2)[1:] * (psi[1:] - psi[:-1])
    vp[:, 1:] = (mV[-1] * hvr / (cu2 * dxt2))[:, 1:] * (psi[:, 1:] - psi[:, :-1])

    def line(k, uu, vv):
        b, d = M.boundary[k, :M.nr_boundary[k]], M.line_dir[k, :M.nr_boundary[k]]
        i, j = (torch.from_numpy(b[:, q].astype(np.int64)).cuda() + 1 for q in (0, 1))
        keep = (i >= 1) & (i <= nx + 1) & (j >= 1) & (j <= ny + 1)
        d = torch.from_numpy(d.astype(np.int64)).cuda()[keep]
        i, j = i[keep], j[keep]
        north, south = uu[j + 1, i] * dxu[i] * cost[j + 1], uu[j, i] * dxu[i] * cost[j]
        west, east = vv[j, i] * dyu[j], vv[j, i + 1] * dyu[j]
        t = torch.zeros_like(north)
        for dd, val in (((1, 0), west + north), ((-1, 0), -east - south), ((0, 1), west - south), ((0, -1), north - east)):
            t = torch.where((d[:, 0] == dd[0]) & (d[:, 1] == dd[1]), val, t)
        return t.sum()

    AB, dt = M.AB_eps, M.dt_mom
    n = M.nisle
    dpsin0 = torch.zeros(n, dtype=torch.float64, device="cuda")
    psi1 = _t(host["psi"][..., 1]) + dt * ((1.5 + AB) * dp1 - (0.5 + AB) * dp0)
    if n > 1:
        rhs = torch.stack([line(k, fpx, fpy) - line(k, up, vp) for k in range(1, n)])
        dpsin0[1:] = torch.linalg.solve(torch.from_numpy(host["line_psin"][1:, 1:].copy()).cuda(), rhs)
        psin, dpsinm = _t(host["psin"]), torch.from_numpy(host["dpsin"][:, 0].copy()).cuda()
        for k in range(1, n):
            psi1 = psi1 + dt * ((1.5 + AB) * dpsin0[k] - (0.5 + AB) * dpsinm[k]) * psin[k]
    # velocities at the new level, their cyclic halo, and w
    new = []
    for q, dq, dqm, mx, mask, hr in ((u, du, _t(host["du"][..., 0]), du_mix, mU, hur),
                                     (v, dv, _t(host["dv"][..., 0]), dv_mix, mV, hvr)):
        x = q + dt * (mx + (1.5 + AB) * dq - (0.5 + AB) * dqm) * mask
        new.append(x - (x * mask * dzt).sum(0) * mask * hr)
    s(new[0])[...] -= s(mU) * (s(psi1) - s(psi1, 0, -1)) / s(dyt2) * s(hur)
    s(new[1])[...] += s(mV) * (s(psi1) - s(psi1, -1)) / (s(cu2) * s(dxt2)) * s(hvr)
    for x in new:
        x[..., :2], x[..., -2:] = x[..., -4:-2].clone(), x[..., 2:4].clone()
    un, vn = new
    wn = _t(host["w"][..., 2]).clone()
    div = (un[:, 1:, 1:] - un[:, 1:, :-1]) / (ct2 * dxt2)[1:, 1:] + (
        (cu2 * vn)[:, 1:, 1:] - (cu2 * vn)[:, :-1, 1:]) / (ct2 * dyt2)[1:, 1:]
    wn[:, 1:, 1:] = -torch.cumsum((mW * dzt)[:, 1:, 1:] * div, 0)
    F3 = lambda a: a.permute(*reversed(range(a.dim())))
    return {"u": F3(un), "v": F3(vn), "w": F3(wn), "psi": F3(psi1), "dpsi": F3(dp1), "du": F3(du), "dv": F3(dv),
            "du_mix": F3(du_mix), "dv_mix": F3(dv_mix), "p_hydro": F3(ph), "dpsin": dpsin0}


def _exact_train(S):
    """Loss and gradient of one training step with the network evaluated in 64 bits throughout."""
    M = S["M"]
    nx, ny = M.nx, M.ny
    op = _operator(M)
    unk = op["unk"].to(torch.float64)
    nu = unk.sum()
    diag = -(op["cw"] + op["ce"] + op["cs"] + op["cn"]) / op["D"]
    r = S["r"].T[2:-2, 2:-2] * unk
    scale = torch.sqrt((r * r).sum() / nu)
    dbar = (diag.abs() * unk).sum() / nu
    hur = _inner(M.hur) * unk
    x = torch.stack([r / scale, unk, hur * nu / hur.sum(), _t(M.cosu)[2:-2][:, None].expand(ny, nx)])
    Hp, Wp = (ny + 7) // 8 * 8, (nx + 7) // 8 * 8
    x = F.pad(x, (0, Wp - nx, 0, Hp - ny))[None]
    x = torch.cat([x, x.new_zeros(1, 12, Hp, Wp)], 1)
    prm = torch.from_numpy(S["net"].get_params().astype(np.float64)).cuda().requires_grad_()
    ws, bs, o = [], [], 0
    for ci, co in learned.LAYERS:
        ws.append(prm[o:o + ci * co * 9].view(co, ci, 3, 3))
        o += ci * co * 9
    for ci, co in learned.LAYERS:
        bs.append(prm[o:o + co])
        o += co
    conv = lambda k, a: F.conv2d(a, ws[k], bs[k], padding=1)
    pool = lambda a: F.avg_pool2d(a, 2)
    up = lambda a: a.repeat_interleave(2, 2).repeat_interleave(2, 3)
    s1 = torch.relu(conv(1, torch.relu(conv(0, x))))
    s2 = torch.relu(conv(3, torch.relu(conv(2, pool(s1)))))
    s3 = torch.relu(conv(5, torch.relu(conv(4, pool(s2)))))
    b4 = torch.relu(conv(7, torch.relu(conv(6, pool(s3)))))
    u3 = torch.relu(up(conv(8, b4)) + s3)
    u2 = torch.relu(up(conv(9, u3)) + s2)
    u1 = torch.relu(up(conv(10, u2)) + s1)
    z = conv(11, u1)[0, 0, :ny, :nx] * unk
    e = S["e"].T[2:-2, 2:-2] * unk * (dbar / scale)
    energy = lambda a: -(a * op["D"] * _apply(op, a)).sum()
    loss = energy(z - e) / energy(e)
    loss.backward()
    return {"loss": float(loss.detach()), "grads": prm.grad}
