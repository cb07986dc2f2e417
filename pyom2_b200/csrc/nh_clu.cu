// Cluster-resident congrad_non_hydro (non_hydrostatic.f90:146-242) for small
// grids: x-z slices and small tanks in one thread-block cluster, with the
// per-cell arithmetic of nh_cg_kernel and the reductions and exchanges of the
// two-dimensional cluster kernel (cg_clu.cuh): tagged words pushed into the
// other blocks' shared memory, no cluster barrier inside the solve.
//
// The grid is cut in x and y; a block holds whole columns of its piece.  A
// thread owns P consecutive levels of one column: residual, direction, A s and
// p_non_hydro in registers, its vertical neighbours' direction mostly too; the
// direction with a one-cell rim in shared memory.  The west, east, south and
// north faces' (residual, direction) travel as tagged records, and the reader
// forms the neighbour's new direction from them as its owner does.
//
// The kernel it replaces for these sizes (one cell per thread in compact order,
// neighbours read from the owners' shared memory in both sweeps, two cluster
// barriers and two 32-warp reductions an iteration) took 7.06 us per iteration
// on a 160 x 1 x 60 slice; this one 2.93 us.
#include <math.h>

#include "cg_clu.cuh"
#include "clu_dev.cuh"
#include "nonhydro.cuh"

namespace pyomgpu {

template <int NT, int P, bool CX, bool CY>
__global__ void __launch_bounds__(NT, 1) nh_clu_kernel(const __grid_constant__ NHParams Pm) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int NW = NT / 32;
  __shared__ double wred[2 * 2 * 2 * NW];
  __shared__ int s_dead[2];
  const NHGeo G = Pm.G;
  const NHOp op = Pm.op;
  const int nx = G.g.nx, ny = G.g.ny, nz = G.nz;
  const int tid = threadIdx.x, rank = (int)clu_rank(), npx = Pm.cnpx, npy = Pm.cnpy, nblk = npx * npy;
  const int px = rank % npx, py = rank / npx;
  const int ilo = 1 + (int)(((long long)px * nx) / npx), ihi = (int)(((long long)(px + 1) * nx) / npx);
  const int jlo = 1 + (int)(((long long)py * ny) / npy), jhi = (int)(((long long)(py + 1) * ny) / npy);
  const int pw = ihi - ilo + 1, ph = jhi - jlo + 1, sp = pw + 2, lv = sp * (ph + 2);
  const int wmax = Pm.cw, hmax = Pm.ch, kp = (nz + P - 1) / P * P;
  // shared memory laid out for the largest piece (an inbox sits at one offset in all blocks); levels padded to
  // whole segments, one level of zeros below and above
  double* ss = reinterpret_cast<double*>(smem);            // [level + 1][row + 1][column + 1]
  double* stT = ss + (size_t)(wmax + 2) * (hmax + 2) * (kp + 2);  // tT, then tB, of the levels
  double* spub = stT + 2 * kp;                             // staged faces: residual, then direction, per entry
  const int nWE = hmax * nz, nSN = wmax * nz, nent = 2 * (nWE + nSN);  // west, east, south, north
  unsigned char* box = reinterpret_cast<unsigned char*>(spub + 2 * (size_t)nent);
  box = smem + (((size_t)(box - smem) + 15) & ~(size_t)15);
  constexpr uint32_t kRec = 32;
  const uint32_t hbox = (uint32_t)__cvta_generic_to_shared(box);
  const CluRed R{hbox + kRec * (uint32_t)nent, wred, nblk, rank, &Pm.ctl->error, Pm.timeout_ns};
  for (int e = tid; e < (wmax + 2) * (hmax + 2) * (kp + 2); e += NT) ss[e] = 0.0;
  for (int k = tid; k < kp; k += NT) {
    stT[k] = k < nz ? op.tT[k] : 0.0;
    stT[kp + k] = k < nz ? op.tB[k] : 0.0;
  }
  {  // tag 0 everywhere: epochs and exchanges count from 1
    unsigned long long* b = reinterpret_cast<unsigned long long*>(box);
    for (int e = tid; e < nent * 4 + 8 * kCluMaxSlots * 2; e += NT) b[e] = 0ull;
    if (tid < 2) s_dead[tid] = 0;
  }
  __syncthreads();  // the initial residual's loop reads the vertical factors of other warps
  const int rW = px > 0 ? rank - 1 : (CX ? rank + npx - 1 : -1), rE = px < npx - 1 ? rank + 1 : (CX ? rank - (npx - 1) : -1);
  const int rS = py > 0 ? rank - npx : (CY ? rank + npx * (npy - 1) : -1);
  const int rN = py < npy - 1 ? rank + npx : (CY ? rank - npx * (npy - 1) : -1);
  const bool halo = rW >= 0 || rE >= 0 || rS >= 0 || rN >= 0;  // the same in every thread of the block

  // this thread's segment: column (lx, ly), levels k0 .. k0+nlev-1 (0-based)
  const int col = tid % (wmax * hmax), lx = col % wmax, ly = col / wmax, k0 = tid / (wmax * hmax) * P;
  const int nlev = (lx < pw && ly < ph && k0 < nz) ? min(P, nz - k0) : 0;
  const int i = ilo + lx, j = jlo + ly;
  const size_t q2 = nlev > 0 ? G.g.at(i, j) : 0;
  const double tE = nlev > 0 ? op.tE[q2] : 0.0, tW = nlev > 0 ? op.tW[q2] : 0.0;
  const double tN = nlev > 0 ? op.tN[j + 1] : 0.0, tS = nlev > 0 ? op.tS[j + 1] : 0.0;
  double s[P], q[P], r[P], x[P];  // direction, A s, residual, p_non_hydro
  double cc[P];                   // centre coefficient, in make_coeff_non_hydro's accumulation order
  uint32_t fl[(P + 3) / 4];       // flag bytes
  auto flag = [&](int u) -> uint32_t { return fl[u / 4] >> (8 * (u % 4)) & 0xffu; };

  // the faces of this thread's segment to their staging entries
  auto stage = [&]() {
    if (nlev == 0) return;
    auto put = [&](int base, int n, int at) {
#pragma unroll
      for (int u = 0; u < P; u++)
        if (u < nlev) {
          const int e = base + (k0 + u) * n + at;
          spub[e] = r[u];
          spub[nent + e] = s[u];
        }
    };
    if (lx == 0 && rW >= 0) put(0, ph, ly);
    if (lx == pw - 1 && rE >= 0) put(nWE, ph, ly);
    if (ly == 0 && rS >= 0) put(2 * nWE, pw, lx);
    if (ly == ph - 1 && rN >= 0) put(2 * nWE + nSN, pw, lx);
  };
  // staged faces to the blocks across them: a west face is the reader's east halo, and so on (blocks that share
  // a face have the same extent along it)
  auto send_halo = [&](unsigned n) {
    auto face = [&](int from, int to, int count, int rk) {
      if (rk < 0) return;
      const uint32_t a = clu_map(hbox + kRec * (uint32_t)to, (uint32_t)rk);
      for (int m = tid; m < count; m += NT) clu_put(a + kRec * (uint32_t)m, spub[from + m], spub[nent + from + m], n);
    };
    face(0, nWE, ph * nz, rW);
    face(nWE, 0, ph * nz, rE);
    face(2 * nWE, 2 * nWE + nSN, pw * nz, rS);
    face(2 * nWE + nSN, 2 * nWE, pw * nz, rN);
  };

  NHCtl ctl;
  unsigned ep = 1, xch = 1;  // reduction, face exchange
  // A thread whose wait ran out says so before the next block barrier, after which all threads of the block
  // leave together; flags of alternate barriers, so none is read while it may be set.
  bool dead = false;
  unsigned nbar = 0;
  auto block_sync = [&]() -> bool {
    if (dead) s_dead[nbar & 1u] = 1;
    __syncthreads();
    return s_dead[nbar++ & 1u] == 0;
  };
  const int kWE = tid / ph, kSN = tid / pw;  // levels of this thread's first records
  // received faces: the neighbours' new direction res + bq s_old (:189) onto the rim; the two faces across one
  // direction hold the same cells, so a thread takes the same record of both (a wait and a division for each face:
  // 160 x 1 x 60 3.11 us per iteration, now 2.93; 48 x 40 x 24 9.08, now 8.56)
  auto recv_halo = [&](double bq, unsigned n) {
    auto faces = [&](int len, int at0, int rim0, int rk0, int at1, int rim1, int rk1, int stride, int kt) {
      if (rk0 < 0 && rk1 < 0) return;
      for (int m = tid; m - tid < len * nz; m += NT) {  // the whole warp polls until all its records are there
        const bool m0 = m < len * nz && rk0 >= 0, m1 = m < len * nz && rk1 >= 0;
        const int k = m == tid ? kt : m / len, o = (k + 1) * lv + (m - k * len) * stride;
        double r0 = 0.0, s0 = 0.0, r1 = 0.0, s1 = 0.0;
        unsigned long long t0 = 0;
        for (unsigned spin = 0; !dead; spin++) {
          bool ok = !m0 || clu_get(hbox + kRec * (uint32_t)(at0 + m), r0, s0, n);
          ok = (!m1 || clu_get(hbox + kRec * (uint32_t)(at1 + m), r1, s1, n)) && ok;
          if (__all_sync(0xffffffffu, ok)) break;
          if (spin == 0) t0 = globaltimer_ns();
          dead = __any_sync(0xffffffffu, clu_expired(R.err, spin + 1, t0, R.tmo));
        }
        if (m0 && !dead) ss[o + rim0] = __dadd_rn(r0, __dmul_rn(bq, s0));
        if (m1 && !dead) ss[o + rim1] = __dadd_rn(r1, __dmul_rn(bq, s1));
      }
    };
    faces(ph, 0, sp, rW, nWE, sp + pw + 1, rE, sp, kWE);
    faces(pw, 2 * nWE, 1, rS, 2 * nWE + nSN, (ph + 1) * sp + 1, rN, 1, kSN);
  };

  bool ns = false;  // a cell of this warp has a south or a north face (an x-z slice has none)
  int how = NHCtl::kGo;
  // ------------------------------------------------------------------ init
  // res = forc - A p (interior), rsold = dot_3D(res, res)  (:163-176)
  {
    double v[2] = {0.0, 0.0};
#pragma unroll
    for (int w = 0; w < (P + 3) / 4; w++) fl[w] = 0;
#pragma unroll
    for (int u = 0; u < P; u++) {
      s[u] = q[u] = r[u] = x[u] = cc[u] = 0.0;
      if (u < nlev) {
        const int k = k0 + u + 1;
        const size_t c = G.at(i, j, k);
        const uint32_t f = __ldg(op.flags + op.fidx(ny, i, j, k));
        const double a = nh_apply(op, G, i, j, k, f, [&](int di, int dj, int dk) {
          return Pm.p[c + (ptrdiff_t)di + (ptrdiff_t)dj * G.g.pitch + (ptrdiff_t)dk * (ptrdiff_t)G.plane];
        });
        const double fo = Pm.forc[(size_t)(i + 1) + (size_t)(nx + 2 * kOnx) *
                                                        ((size_t)(j + 1) + (size_t)(ny + 2 * kOnx) * (size_t)(k - 1))];
        r[u] = __dsub_rn(fo, a);
        x[u] = Pm.p[c];
        fl[u / 4] |= f << (8 * (u % 4));
        cc[u] = nh_centre(f, tE, tW, tN, tS, stT[k0 + u], stT[kp + k0 + u]);
        if (f & kNHMaskT) {
          v[0] += r[u] * r[u];
          v[1] += fo * fo;
        }
      }
    }
    uint32_t any = 0;
#pragma unroll
    for (int w = 0; w < (P + 3) / 4; w++) any |= fl[w];
    ns = __any_sync(0xffffffffu, any & (kNHN | kNHS) * 0x01010101u);
    stage();
    clu_sync();  // every inbox is cleared, the faces staged
    send_halo(xch);
    clu_send<NW, false>(v[0], v[1], ep, 0, R, Pm.stall_extra != 0);
    dead = !clu_recv<NW, false>(v[0], v[1], ep, 0, R, Pm.stall_extra != 0);
    how = ctl.start(v[0], v[1], Pm);
  }

  while (how == NHCtl::kGo && !dead) {
    // ------------------------------------------------ sweep A: direction, A s
    {
      const double bq = ctl.bq;
      double* o = ss + (k0 + 1) * lv + (ly + 1) * sp + lx + 1;
#pragma unroll
      for (int u = 0; u < P; u++) {
        s[u] = __dadd_rn(r[u], __dmul_rn(bq, s[u]));
        if (u < nlev) o[u * lv] = s[u];
      }
      if (halo) recv_halo(bq, xch++);
    }
    if (!block_sync()) goto out;
    double vA[2] = {0.0, 0.0};  // (s, As), max|s| over maskT
    if (nlev > 0) {
      const double* o = ss + (k0 + 1) * lv + (ly + 1) * sp + lx + 1;
      const double below = o[-lv], above = o[nlev * lv];
      // nh_row term by term over the segment, with selects and the centre coefficient kept: its tests as branches
      // ran one level after the other (8 levels a thread: 240 x 1 x 80 in 4.76 us per iteration, now 3.99; one
      // block, 64 x 1 x 24: 2.52, now 1.69; 160 x 1 x 60 with 4 levels: 3.20, now 3.10)
      auto term = [&](uint32_t face, auto coef, auto val) {
#pragma unroll
        for (int u = 0; u < P; u++) {  // no face beyond the segment's last level: A s = 0 there
          const double n = __dadd_rn(q[u], __dmul_rn(coef(u), val(u)));
          q[u] = (flag(u) & face) ? n : q[u];
        }
      };
#pragma unroll
      for (int u = 0; u < P; u++) q[u] = 0.0;
      term(kNHB, [&](int u) { return stT[kp + k0 + u]; }, [&](int u) { return u > 0 ? s[u > 0 ? u - 1 : 0] : below; });
      if (ns) term(kNHS, [&](int) { return tS; }, [&](int u) { return o[u * lv - sp]; });
      term(kNHW, [&](int) { return tW; }, [&](int u) { return o[u * lv - 1]; });
#pragma unroll
      for (int u = 0; u < P; u++) q[u] = __dadd_rn(q[u], __dmul_rn(cc[u], s[u]));
      term(kNHE, [&](int) { return tE; }, [&](int u) { return o[u * lv + 1]; });
      if (ns) term(kNHN, [&](int) { return tN; }, [&](int u) { return o[u * lv + sp]; });
      term(kNHT, [&](int u) { return stT[k0 + u]; },
           [&](int u) { return u + 1 == nlev ? above : s[u + 1 < P ? u + 1 : u]; });
#pragma unroll
      for (int u = 0; u < P; u++) {
        const bool wet = flag(u) & kNHMaskT;
        vA[0] += wet ? s[u] * q[u] : 0.0;
        vA[1] = fmax(vA[1], wet ? fabs(s[u]) : 0.0);
      }
    }
    ++ep;
    clu_send<NW, true>(vA[0], vA[1], ep, 0, R, false);
    dead = !clu_recv<NW, true>(vA[0], vA[1], ep, 0, R, false);
    if (dead) break;
    double alpha = 0.0;
    how = ctl.after_a(vA[0], vA[1], alpha);
    if (how != NHCtl::kGo) break;
    // ------------------------------------------------ sweep B: residual, p
    double vB[2] = {0.0, 0.0};
#pragma unroll
    for (int u = 0; u < P; u++) {
      r[u] = __dsub_rn(r[u], __dmul_rn(alpha, q[u]));  // res = res - alpha*Ap (:188)
      vB[0] += (flag(u) & kNHMaskT) ? r[u] * r[u] : 0.0;
    }
    ++ep;
    clu_send<NW, false>(vB[0], vB[1], ep, 0, R, false);
    if (halo) {  // the faces for the next direction, while the partial sums travel
      stage();
      if (!block_sync()) goto out;
      send_halo(xch);
    }
#pragma unroll
    for (int u = 0; u < P; u++) x[u] = __dadd_rn(x[u], __dmul_rn(alpha, s[u]));  // :187
    dead = !clu_recv<NW, false>(vB[0], vB[1], ep, 0, R, false);
    if (dead) break;
    how = ctl.after_b(vB[0], alpha);
  }
  if (!block_sync()) goto out;
  ctl.finish(how, Pm.out);
#pragma unroll
  for (int u = 0; u < P; u++)
    if (u < nlev) {
      // p += alpha*s over the whole array: a cyclic halo copy keeps the difference to its cell that it came in with
      double* p = Pm.p + G.at(i, j, k0 + u + 1);
      const double was = *p;
      const ptrdiff_t ox = CX ? (i <= kOnx ? (ptrdiff_t)nx : (i > nx - kOnx ? -(ptrdiff_t)nx : 0)) : 0;
      const ptrdiff_t oy = CY ? (j <= kOnx ? (ptrdiff_t)ny : (j > ny - kOnx ? -(ptrdiff_t)ny : 0)) * G.g.pitch : 0;
      if (ox) p[ox] = x[u] + (p[ox] - was);
      if (oy) p[oy] = x[u] + (p[oy] - was);
      if (ox && oy) p[ox + oy] = x[u] + (p[ox + oy] - was);
      *p = x[u];
    }
out:
  clu_sync();
}

template <int NT, int P>
static const void* nh_clu_ptr(bool cx, bool cy) {
  if (cx) return cy ? (const void*)nh_clu_kernel<NT, P, true, true> : (const void*)nh_clu_kernel<NT, P, true, false>;
  return cy ? (const void*)nh_clu_kernel<NT, P, false, true> : (const void*)nh_clu_kernel<NT, P, false, false>;
}
const void* nh_clu_kernel_ptr(int nt, int p, bool cx, bool cy) {
  switch (nt * 100 + p) {
    case 12804: return nh_clu_ptr<128, 4>(cx, cy);
    case 12808: return nh_clu_ptr<128, 8>(cx, cy);
    case 25604: return nh_clu_ptr<256, 4>(cx, cy);
    case 25608: return nh_clu_ptr<256, 8>(cx, cy);
    case 25612: return nh_clu_ptr<256, 12>(cx, cy);
    default: return nullptr;
  }
}

}  // namespace pyomgpu
