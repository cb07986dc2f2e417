// Cluster-resident Jacobi-PCG for small grids: congrad_streamfunction
// (solve_streamfct.f90:153-327) and congrad_surf_press (solve_pressure.f90:
// 137-249) with the arithmetic and control flow of the resident kernel
// (cg_res.cu), whole grid in one thread-block cluster of at most 16 blocks.
//
// What bounds a small solve is the two reductions of an iteration, not its
// points: across the whole chip each costs an L2 round trip of ~2 us, so a
// 40 x 40 grid took 4.6 us per iteration on ten SMs.  Inside a cluster the same
// words go straight into the other blocks' shared memory:
//   * a block's partial sums are pushed, as tagged words (cg_ctl.cuh), into the
//     inbox of every block of the cluster; every warp polls its own block's
//     inbox, sums the slots in a fixed order and runs the control step itself,
//     so a decision needs no second block barrier (a block alone in its
//     cluster reads its warps' partials instead);
//   * the boundary values (Z res, direction) go from the owning thread's
//     registers into the neighbour's inbox, in the sweep that makes them;
//   * all warps (four or eight a block) own points, column segments of P rows
//     as in cg_res.cu: residual, direction, Z*res (or A s), solution and Z in
//     registers, the face couplings too up to P = 4, else in shared memory.
// An inbox word is rewritten only after every reader has passed it: a slot of
// epoch e at e+2, when every block has published e+1; a halo record one
// iteration later, when its reader has published the sweep A in between.
// Every wait is bounded by %globaltimer; a block that gives up still meets the
// cluster's last barrier, so no block's shared memory goes away under a
// neighbour's store.
#include <math.h>

#include "cg_clu.cuh"
#include "cg_ctl.cuh"
#include "clu_dev.cuh"

namespace pyomgpu {
template <typename T, int NT, int P, bool SP>
__global__ void __launch_bounds__(NT, 1) cg_clu_kernel(const __grid_constant__ CGResParams Pm) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int NW = NT / 32;
  __shared__ double wred[2 * 2 * 2 * NW];
  __shared__ int s_dead[2];
  const Geo g = Pm.g;
  const OpDev<T> op = res_op<T>(Pm);
  const int tid = threadIdx.x, rank = (int)clu_rank(), nblk = Pm.npx * Pm.npy;
  const int px = rank % Pm.npx, py = rank / Pm.npx;
  const int ilo = 1 + (int)(((long long)px * g.nx) / Pm.npx), ihi = (int)(((long long)(px + 1) * g.nx) / Pm.npx);
  const int jlo = 1 + (int)(((long long)py * g.ny) / Pm.npy), jhi = (int)(((long long)(py + 1) * g.ny) / Pm.npy);
  const int pw = ihi - ilo + 1, ph = jhi - jlo + 1, sp = pw + 2;
  const int wmax = Pm.wmax, hmax = Pm.hmax, hp = (hmax + P - 1) / P * P;
  // Every block lays its shared memory out for the largest piece, so an inbox sits at one offset in all of
  // them; rows are padded to whole column segments with zero coefficients, so the sweeps run over all P rows of
  // a segment without a branch per point (with one, the points' chains ran one after another: 140 cycles each).
  T* ss = reinterpret_cast<T*>(smem);       // (pw+2) x (hp+2): direction, halo included
  T* sfx = ss + (wmax + 2) * (hp + 2);      // (pw+1) x hp: FX(ilo+lx, j)
  T* sfy = sfx + (wmax + 1) * hp;           // pw x (hp+1): FY(i, jlo+ly)
  T* sbx = sfy + wmax * (hp + 1);           // bx, then by, of the rows
  T* spub = sbx + 2 * hp;                   // staged boundary values: Z res, then direction, per entry
  const int nent = 2 * (wmax + hmax);       // entries: west, east (hmax each), south, north (wmax each)
  unsigned char* box = smem + (sizeof(T) * clu_fields(wmax, hp, nent) + 15) / 16 * 16;
  constexpr uint32_t kRec = 4 * (uint32_t)sizeof(T);  // bytes of a halo record
  const uint32_t hbox = (uint32_t)__cvta_generic_to_shared(box);
  const CluRed R{hbox + kRec * (uint32_t)nent, wred, nblk, rank, &Pm.ctl->error, Pm.timeout_ns};

  {
    const int nf = (int)clu_fields(wmax, hp, nent);
    for (int e = tid; e < nf; e += NT) ss[e] = (T)0;
    // tag 0 everywhere: epochs and exchanges count from 1
    const int words = nent * (int)(kRec / 8) + 8 * kCluMaxSlots * 2;
    unsigned long long* b = reinterpret_cast<unsigned long long*>(box);
    for (int e = tid; e < words; e += NT) b[e] = 0ull;
    if (tid < 2) s_dead[tid] = 0;
  }
  __syncthreads();
  for (int e = tid; e < (pw + 1) * ph; e += NT) sfx[e] = op.FX[g.at(ilo + e % (pw + 1), jlo + e / (pw + 1))];
  for (int e = tid; e < pw * (ph + 1); e += NT) sfy[e] = op.FY[g.at(ilo + e % pw, jlo + e / pw)];
  for (int e = tid; e < ph; e += NT) {
    sbx[e] = op.bx[jlo + e + 1];
    sbx[hp + e] = op.by[jlo + e + 1];
  }

  // neighbours (rank, or -1 at a closed edge); the boundary entries this thread sends, and the halo entries it
  // receives: a west entry of one block is an east halo entry of the block across the edge, and so on
  const int rW = px > 0 ? rank - 1 : (g.cyclic_x ? rank + Pm.npx - 1 : -1);
  const int rE = px < Pm.npx - 1 ? rank + 1 : (g.cyclic_x ? rank - (Pm.npx - 1) : -1);
  const int rS = py > 0 ? rank - Pm.npx : (g.cyclic_y ? rank + Pm.npx * (Pm.npy - 1) : -1);
  const int rN = py < Pm.npy - 1 ? rank + Pm.npx : (g.cyclic_y ? rank - Pm.npx * (Pm.npy - 1) : -1);
  const bool halo = rW >= 0 || rE >= 0 || rS >= 0 || rN >= 0;  // the same in every thread of the block
  int hs[2];                 // index of the halo point in ss, -1: none
  uint32_t hr[2], hd[2];     // address of its record here; record in the neighbour's inbox of the entry sent
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int h = tid + e * NT;
    hs[e] = -1;
    hr[e] = hbox + kRec * (uint32_t)h;
    hd[e] = 0;
    int to = -1, at = 0;
    if (h < hmax) {
      if (h < ph && rW >= 0) {
        hs[e] = (h + 1) * sp;
        to = rW;
        at = hmax + h;
      }
    } else if (h < 2 * hmax) {
      if (h - hmax < ph && rE >= 0) {
        hs[e] = (h - hmax + 1) * sp + pw + 1;
        to = rE;
        at = h - hmax;
      }
    } else if (h < 2 * hmax + wmax) {
      if (h - 2 * hmax < pw && rS >= 0) {
        hs[e] = h - 2 * hmax + 1;
        to = rS;
        at = h + wmax;
      }
    } else if (h < nent) {
      if (h - 2 * hmax - wmax < pw && rN >= 0) {
        hs[e] = (ph + 1) * sp + h - 2 * hmax - wmax + 1;
        to = rN;
        at = h - wmax;
      }
    }
    if (to >= 0) hd[e] = clu_map(hbox + kRec * (uint32_t)at, (uint32_t)to);
  }

  // this thread's column segment: column lx, rows ly0 .. ly0+nrow-1
  const int lx = tid % wmax, ly0 = (tid / wmax) * P;
  const int nrow = (lx < pw && ly0 < ph) ? min(P, ph - ly0) : 0;
  const int i = ilo + lx;
  const T axi = nrow > 0 ? op.ax[i + 1] : (T)0;
  T s[P], q[P], r[P], x[P], z[SP ? 1 : P];  // direction; Z res, then A s; residual; solution; Z
  unsigned wbits = 0;                       // SP: maskT
  // The sweeps are bound by shared-memory reads (six doubles a point: 1030 cycles for the 1600 points of a
  // 40 x 40 grid in one block), so short segments keep their face couplings in registers.
  constexpr bool kRegC = P <= 4;
  T cw[kRegC ? P : 1], ce[kRegC ? P : 1], cy[kRegC ? P + 1 : 1];
  // boundary values of this thread's points to the staging entries
  auto stage = [&]() {
    if (nrow == 0) return;
    const bool w = lx == 0 && rW >= 0, e = lx == pw - 1 && rE >= 0;
    if (w || e) {  // pieces are at least two columns wide
      const int c = (w ? 0 : hmax) + ly0;
#pragma unroll
      for (int u = 0; u < P; u++)
        if (u < nrow) {
          spub[c + u] = q[u];
          spub[nent + c + u] = s[u];
        }
    }
    if (ly0 == 0) {
      spub[2 * hmax + lx] = q[0];
      spub[nent + 2 * hmax + lx] = s[0];
    }
    if (ly0 + nrow == ph) {
      T ql = q[0], sl = s[0];  // the last row's, by selects (an index would move q and s to local memory)
#pragma unroll
      for (int u = 1; u < P; u++) {
        ql = u < nrow ? q[u] : ql;
        sl = u < nrow ? s[u] : sl;
      }
      spub[2 * hmax + wmax + lx] = ql;
      spub[nent + 2 * hmax + wmax + lx] = sl;
    }
  };
  // staged entries to the blocks across the edges, one or two a thread, exchange number n
  auto send_halo = [&](unsigned n) {
#pragma unroll
    for (int e = 0; e < 2; e++)
      if (hs[e] >= 0) clu_put(hd[e], spub[tid + e * NT], spub[nent + tid + e * NT], n);
  };

  ResCtl C;
  unsigned ep = 1;   // reduction
  unsigned xch = 1;  // halo exchange
  bool stopped = false;
  // A thread whose wait ran out says so before the next block barrier, after which all threads of the block
  // leave together; flags of alternate barriers, so none is read while it may be set.
  bool dead = false;
  unsigned nbar = 0;
  auto block_sync = [&]() -> bool {
    if (dead) s_dead[nbar & 1u] = 1;
    __syncthreads();
    return s_dead[nbar++ & 1u] == 0;
  };
  // ------------------------------------------------------------------ init
  // res = forc - A sol, solve_streamfct.f90:196-201 / solve_pressure.f90:163-168
  {
    double v[4] = {0.0, 0.0, 0.0, 0.0};  // beta, bb, rr, zresmax
#pragma unroll
    for (int u = 0; u < P; u++) {
      s[u] = q[u] = r[u] = x[u] = (T)0;
      if (!SP) z[SP ? 0 : u] = (T)0;
      if (u < nrow) {
        const int j = jlo + ly0 + u;
        const T f = res_forc<T>(Pm)[sizeof(T) == 8 ? fidx(g.nx, i, j) : g.at(i, j)];
        const T rv = f - apply_point(op, g, (const T*)res_solv<T>(Pm), i, j);
        const T w = op.W[g.at(i, j)];
        const T zr = SP ? rv : w * rv;
        if constexpr (SP) {  // multiplied by the weight, so a NaN on land spreads as in the reference
          wbits |= w != (T)0 ? 1u << u : 0u;
          v[0] += (double)rv * (double)rv * (double)w;
          v[1] += (double)f * (double)f * (double)w;
        } else {
          v[0] += (double)zr * (double)rv;
          if (w != (T)0) {
            v[1] += (double)f * (double)f;
            v[2] += (double)rv * (double)rv;
          }
          v[3] = fmax(v[3], fabs((double)zr));
          z[SP ? 0 : u] = w;
        }
        r[u] = rv;
        q[u] = zr;
        x[u] = res_solv<T>(Pm)[g.at(i, j)];
      }
    }
    stage();
    clu_sync();  // every inbox is cleared, every shared field loaded, the boundary staged
    if constexpr (kRegC) {
      const int fx0 = nrow > 0 ? ly0 * (pw + 1) + lx : 0, fy0 = nrow > 0 ? ly0 * pw + lx : 0;
      cy[0] = sfy[fy0];
#pragma unroll
      for (int u = 0; u < P; u++) {
        cw[u] = sfx[fx0 + u * (pw + 1)];
        ce[u] = sfx[fx0 + u * (pw + 1) + 1];
        cy[u + 1] = sfy[fy0 + (u + 1) * pw];
      }
    }
    send_halo(xch);
    clu_send<NW, false>(v[0], v[1], ep, 0, R, Pm.stall_extra != 0);
    clu_send<NW, true>(v[2], v[3], ep, 1, R, Pm.stall_extra != 0);
    dead = !clu_recv<NW, false>(v[0], v[1], ep, 0, R, Pm.stall_extra != 0);
    if (!dead) dead = !clu_recv<NW, true>(v[2], v[3], ep, 1, R, Pm.stall_extra != 0);
    if constexpr (SP)
      ctl_init_sp(C, Pm, v);
    else
      ctl_init(C, Pm, v);
  }

  while (C.act == kRun && !dead) {
    // ------------------------------------------------ sweep A: direction, As
    {
      const T bq = (T)C.bq;
      T* o = ss + (ly0 + 1) * sp + lx + 1;
#pragma unroll
      for (int u = 0; u < P; u++) {
        s[u] = q[u] + bq * s[u];
        if (u < nrow) o[u * sp] = s[u];
      }
      if (halo) {  // the whole warp polls until all its records are there (see warp_sum_mma)
        T hq[2], hd2[2];
        unsigned long long t0 = 0;
        for (unsigned spin = 0;; spin++) {
          bool ok = true;
#pragma unroll
          for (int e = 0; e < 2; e++)
            if (hs[e] >= 0) ok = clu_get(hr[e], hq[e], hd2[e], xch) && ok;
          if (__all_sync(0xffffffffu, ok)) break;
          if (spin == 0) t0 = globaltimer_ns();
          if (__any_sync(0xffffffffu, clu_expired(R.err, spin + 1, t0, R.tmo))) {
            dead = true;
            break;
          }
        }
#pragma unroll
        for (int e = 0; e < 2; e++)
          if (hs[e] >= 0 && !dead) ss[hs[e]] = hq[e] + bq * hd2[e];
      }
      xch++;
    }
    if (!block_sync()) goto out;
    double vA[2] = {0.0, 0.0};  // (s, As), max|s|
    if (nrow > 0) {
      const T* o = ss + (ly0 + 1) * sp + lx + 1;
      const T *fx = sfx + ly0 * (pw + 1) + lx, *fy = sfy + ly0 * pw + lx, *bx = sbx + ly0, *by = sbx + hp + ly0;
      const T below = o[-sp], above = o[nrow * sp];  // the rows past the segment's ends
      T fys = kRegC ? cy[0] : fy[0];
#pragma unroll
      for (int u = 0; u < P; u++) {
        const T sc = s[u];
        const T se = o[u * sp + 1], sw = o[u * sp - 1];
        const T sn = u + 1 == nrow ? above : s[u + 1 < P ? u + 1 : u];
        const T so = (u > 0) ? s[u > 0 ? u - 1 : 0] : below;
        const T fxw = kRegC ? cw[kRegC ? u : 0] : fx[u * (pw + 1)], fxe = kRegC ? ce[kRegC ? u : 0] : fx[u * (pw + 1) + 1];
        const T fyn = kRegC ? cy[kRegC ? u + 1 : 0] : fy[(u + 1) * pw];
        T a = axi * bx[u] * (fxe * (se - sc) + fxw * (sw - sc)) + by[u] * (fyn * (sn - sc) + fys * (so - sc));
        fys = fyn;
        if constexpr (SP) {
          const bool wet = wbits >> u & 1u;
          a += (wet ? op.dcoef : (T)0) * sc;
          vA[0] += u < nrow ? (double)sc * (double)a * (wet ? 1.0 : 0.0) : 0.0;
          vA[1] = fmax(vA[1], wet ? fabs((double)sc) : 0.0);
        } else {
          vA[0] += u < nrow ? (double)sc * (double)a : 0.0;
          vA[1] = fmax(vA[1], u < nrow ? fabs((double)sc) : 0.0);
        }
        q[u] = a;
      }
    }
    ++ep;
    clu_send<NW, true>(vA[0], vA[1], ep, 0, R, false);
    dead = !clu_recv<NW, true>(vA[0], vA[1], ep, 0, R, false);
    if (dead) break;
    if constexpr (SP)
      ctl_after_a_sp(C, Pm, vA);
    else
      ctl_after_a(C, Pm, vA);
    if (C.act != kRun) break;
    // ---------------------------------------------- sweep B: residual update
    const T alpha = (T)C.alpha;
    double vB[2] = {0.0, 0.0};  // (Z res, res), sum res^2 over the unknowns
#pragma unroll
    for (int u = 0; u < P; u++) {
      const T rv = r[u] - alpha * q[u];
      r[u] = rv;
      if constexpr (SP) {
        vB[0] += u < nrow ? (double)rv * (double)rv * ((wbits >> u & 1u) ? 1.0 : 0.0) : 0.0;
        q[u] = rv;
      } else {
        const T w = z[SP ? 0 : u];
        const T zr = w * rv;
        vB[0] += u < nrow ? (double)zr * (double)rv : 0.0;
        vB[1] += w != (T)0 ? (double)rv * (double)rv : 0.0;
        q[u] = zr;
      }
    }
    ++ep;
    if (!C.stop_after) {
      clu_send<NW, false>(vB[0], vB[1], ep, 0, R, false);
      if (halo) {  // the boundary values for the next direction, while the partial sums travel
        stage();
        if (!block_sync()) goto out;
        send_halo(xch);
      }
    }
    // sol += alpha*s (solve_streamfct.f90:278)
#pragma unroll
    for (int u = 0; u < P; u++) x[u] = x[u] + alpha * s[u];
    if (C.stop_after) {
      stopped = true;
      break;
    }
    dead = !clu_recv<NW, false>(vB[0], vB[1], ep, 0, R, false);
    if (dead) break;
    if constexpr (SP)
      ctl_after_b_sp(C, vB);
    else
      ctl_after_b(C, Pm, vB);
  }
  if (!block_sync()) goto out;
  if (rank == 0 && tid == 0) {
    const int converged = stopped || C.act == kDoneOk;
    Pm.out->iterations = C.n;
    Pm.out->converged = converged;
    Pm.out->status = converged ? PYOMGPU_OK : (C.est != C.est ? PYOMGPU_NAN : C.status);
    Pm.out->est = C.est;
  }
#pragma unroll
  for (int u = 0; u < P; u++)
    if (u < nrow) res_solv<T>(Pm)[g.at(i, jlo + ly0 + u)] = x[u];
out:
  clu_sync();
}

template <typename T, bool SP>
static const void* clu_ptr(int nt, int p) {
  switch (nt * 100 + p) {
    case 12804: return (const void*)cg_clu_kernel<T, 128, 4, SP>;
    case 12806: return (const void*)cg_clu_kernel<T, 128, 6, SP>;
    case 12808: return (const void*)cg_clu_kernel<T, 128, 8, SP>;
    case 12812: return (const void*)cg_clu_kernel<T, 128, 12, SP>;
    case 25604: return (const void*)cg_clu_kernel<T, 256, 4, SP>;
    case 25606: return (const void*)cg_clu_kernel<T, 256, 6, SP>;
    case 25608: return (const void*)cg_clu_kernel<T, 256, 8, SP>;
    case 25612: return (const void*)cg_clu_kernel<T, 256, 12, SP>;
    default: return nullptr;
  }
}

const void* cg_clu_kernel_ptr(int nt, int p, bool surf_press, bool fp32) {
  if (surf_press) return fp32 ? nullptr : clu_ptr<double, true>(nt, p);
  return fp32 ? clu_ptr<float, false>(nt, p) : clu_ptr<double, false>(nt, p);
}

}  // namespace pyomgpu
