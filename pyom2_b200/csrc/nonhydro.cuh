// Non-hydrostatic pressure operator (non_hydrostatic.f90:70-138, 247-276) in
// compact device form.
//
// make_coeff_non_hydro stores a 3x3x3 stencil per cell (27 doubles), of which
// at most seven entries are nonzero: the six faces and the centre.  Every face
// coefficient is a 0/1 face mask times a metric factor that depends on one or
// two of (i, j, k) only:
//
//   east   maskU(i,j,k)   * tE(i,j) = ((1/dxu(i)  )/dxt(i))/cost(j)**2
//   west   maskU(i-1,j,k) * tW(i,j) = ((1/dxu(i-1))/dxt(i))/cost(j)**2
//   north  maskV(i,j,k)   * tN(j)   = (((1/dyu(j)  )/dyt(j))*cosu(j)  )/cost(j)
//   south  maskV(i,j-1,k) * tS(j)   = (((1/dyu(j-1))/dyt(j))*cosu(j-1))/cost(j)
//   top    maskW(i,j,k)   * tT(k)   = (1/dzw(k)  )/dzt(k)      (k < nz)
//   bottom maskW(i,j,k-1) * tB(k)   = (1/dzw(k-1))/dzt(k)      (k > 1)
//
// (mp/a/b/c with mp = 1 rounds exactly like 1/a/b/c, and with mp = 0 gives 0.)
// The device keeps one flag byte per cell (the six face masks and maskT) plus
// the 2-D tables tE, tW and the 1-D tables tN, tS, tT, tB, i.e. 1 byte per
// cell instead of 216.  The centre coefficient is rebuilt in the order the
// reference accumulates it (east, west, north, south, top, bottom), and the
// products are summed in apply_op_3D's (kk, jj, ii) order with separately
// rounded multiplies and adds, so A p is bit-identical to the reference's.
#pragma once
#include <math.h>

#include "cg_clu.cuh"
#include <cuda.h>
#include <stdint.h>

#include "common.cuh"

namespace pyomgpu {

constexpr int kNHThreads = 256;

enum : uint32_t { kNHE = 1u, kNHW = 2u, kNHN = 4u, kNHS = 8u, kNHT = 16u, kNHB = 32u, kNHMaskT = 64u };

// Padded 3-D layout: level k (1..nz) is a padded 2-D field of the Geo layout.
struct NHGeo {
  Geo g;
  int nz;
  size_t plane;  // g.size()
  __host__ __device__ __forceinline__ size_t at(int i, int j, int k) const {
    return (size_t)(k - 1) * plane + g.at(i, j);
  }
  __host__ __device__ __forceinline__ size_t size() const { return plane * (size_t)nz; }
};

struct NHOp {
  const uint8_t* flags;  // [nz][ny][fx], cell (i,j,k) at ((k-1)*ny + j-1)*fx + i-1
  const double* tE;      // padded 2-D
  const double* tW;      // padded 2-D
  const double* tN;      // [ny+4], index j+1
  const double* tS;      // [ny+4], index j+1
  const double* tT;      // [nz], index k-1
  const double* tB;      // [nz], index k-1
  int fx;                // flag row pitch, nx rounded up to 32
  __host__ __device__ __forceinline__ size_t fidx(int ny, int i, int j, int k) const {
    return ((size_t)(k - 1) * (size_t)ny + (size_t)(j - 1)) * (size_t)fx + (size_t)(i - 1);
  }
};

// Centre coefficient of a cell's row (make_coeff_non_hydro's accumulation order).
__device__ __forceinline__ double nh_centre(uint32_t f, double tE, double tW, double tN, double tS, double tT, double tB) {
  double c = 0.0;
  if (f & kNHE) c = __dsub_rn(c, tE);
  if (f & kNHW) c = __dsub_rn(c, tW);
  if (f & kNHN) c = __dsub_rn(c, tN);
  if (f & kNHS) c = __dsub_rn(c, tS);
  if (f & kNHT) c = __dsub_rn(c, tT);
  if (f & kNHB) c = __dsub_rn(c, tB);
  return c;
}
// Operator row with the seven field values given: bottom, south, west,
// centre, east, north, top; t* are the face factors (read only where the
// face flag is set).
__device__ __forceinline__ double nh_row(uint32_t f, double tE, double tW, double tN, double tS, double tT, double tB,
                                         double vb, double vs, double vw, double vc, double ve, double vn, double vt) {
  const double c = nh_centre(f, tE, tW, tN, tS, tT, tB);
  // apply_op_3D: kk outermost, then jj, then ii; zero coefficients add nothing
  double a = 0.0;
  if (f & kNHB) a = __dadd_rn(a, __dmul_rn(tB, vb));
  if (f & kNHS) a = __dadd_rn(a, __dmul_rn(tS, vs));
  if (f & kNHW) a = __dadd_rn(a, __dmul_rn(tW, vw));
  a = __dadd_rn(a, __dmul_rn(c, vc));
  if (f & kNHE) a = __dadd_rn(a, __dmul_rn(tE, ve));
  if (f & kNHN) a = __dadd_rn(a, __dmul_rn(tN, vn));
  if (f & kNHT) a = __dadd_rn(a, __dmul_rn(tT, vt));
  return a;
}

// Operator row of cell (i,j,k) applied to a field given by fetch(di, dj, dk).
template <class Fetch>
__device__ __forceinline__ double nh_apply(const NHOp& op, const NHGeo& G, int i, int j, int k, uint32_t f,
                                           const Fetch& fetch) {
  const size_t q2 = G.g.at(i, j);  // the tables are read-only for the life of the operator
  const double tE = (f & kNHE) ? __ldg(op.tE + q2) : 0.0;
  const double tW = (f & kNHW) ? __ldg(op.tW + q2) : 0.0;
  const double tN = (f & kNHN) ? __ldg(op.tN + j + 1) : 0.0;
  const double tS = (f & kNHS) ? __ldg(op.tS + j + 1) : 0.0;
  const double tT = (f & kNHT) ? __ldg(op.tT + k - 1) : 0.0;
  const double tB = (f & kNHB) ? __ldg(op.tB + k - 1) : 0.0;
  return nh_row(f, tE, tW, tN, tS, tT, tB, (f & kNHB) ? fetch(0, 0, -1) : 0.0, (f & kNHS) ? fetch(0, -1, 0) : 0.0,
                (f & kNHW) ? fetch(-1, 0, 0) : 0.0, fetch(0, 0, 0), (f & kNHE) ? fetch(1, 0, 0) : 0.0,
                (f & kNHN) ? fetch(0, 1, 0) : 0.0, (f & kNHT) ? fetch(0, 0, 1) : 0.0);
}

// setcyclic_xyz (parallel_none.f90) applied per level: store v at (i,j,k) and
// at the halo copies of (i,j) on that level.
template <typename T>
__device__ __forceinline__ void nh_store_cyclic(T* __restrict__ a, const NHGeo& G, int i, int j, int k, T v) {
  store_cyclic(a + (size_t)(k - 1) * G.plane, G.g, i, j, v);
}
template <typename T>
__device__ __forceinline__ void nh_add_cyclic(T* __restrict__ a, const NHGeo& G, int i, int j, int k, T d) {
  add_cyclic(a + (size_t)(k - 1) * G.plane, G.g, i, j, d);
}

struct CGResult;

// Bricks of the CG sweeps: 32 cells in i (one per lane) x ty in j x kc in k,
// kc = (8/ty) * kw.  Warp w works on row jj = w % ty and marches over kw
// levels from (w / ty) * kw.  Per brick and pipeline stage, shared memory
// holds two boxes (brick + one-cell halo: i0-2..i0+33, i.e. 36 doubles
// starting on a 16-byte boundary of the padded layout, j0-1..j0+ty,
// k0-1..k0+kc) -- sweep A: res and s; sweep B: s and, in the second box's
// place, the brick's res and p -- and the brick's flag bytes.
constexpr int kNHBoxX = 36;
__host__ __device__ constexpr size_t nh_al(size_t b) { return (b + 127) / 128 * 128; }
__host__ __device__ constexpr size_t nh_rs_bytes(int ty, int kc) { return (size_t)kNHBoxX * (ty + 2) * (kc + 2) * 8; }
__host__ __device__ constexpr size_t nh_p_bytes(int ty, int kc) { return (size_t)32 * ty * kc * 8; }
__host__ __device__ constexpr size_t nh_f_bytes(int ty, int kc) { return (size_t)32 * ty * kc; }
// stage layout: [box 0][region 1: box 1, or the brick's res then p][flags]
__host__ __device__ constexpr size_t nh_region1_bytes(int ty, int kc) {
  return nh_al(nh_rs_bytes(ty, kc)) > 2 * nh_al(nh_p_bytes(ty, kc)) ? nh_al(nh_rs_bytes(ty, kc))
                                                                       : 2 * nh_al(nh_p_bytes(ty, kc));
}
__host__ __device__ constexpr size_t nh_flags_off(int ty, int kc) {
  return nh_al(nh_rs_bytes(ty, kc)) + nh_region1_bytes(ty, kc);
}
__host__ __device__ constexpr size_t nh_stage_bytes(int ty, int kc) {
  return nh_flags_off(ty, kc) + nh_al(nh_f_bytes(ty, kc));
}
// ns pipeline stages (2..4) + a full and an empty mbarrier per stage
constexpr int kNHMaxStages = 4;
__host__ __device__ constexpr size_t nh_smem_bytes(int ty, int kc, int ns) {
  return (size_t)ns * nh_stage_bytes(ty, kc) + 128;
}
constexpr size_t kNHSmemMax = 220 * 1024;

struct alignas(64) NHParams {
  CUtensorMap map_res, map_s[2];     // 3-D (pitch, ny+4, nz) maps, box 36 x (ty+2) x (kc+2)
  CUtensorMap map_res_brick;         // the same array as map_res, box 32 x ty x kc
  CUtensorMap map_p;                 // 3-D (pitch, ny+4, nz) map of p, box 32 x ty x kc
  CUtensorMap map_f;                 // 3-D (fx, ny, nz) map of the flags, box 32 x ty x kc
  NHGeo G;
  NHOp op;
  int ty, kw, kc;                    // brick shape
  int ns;                            // pipeline stages
  int small_chunk;                   // compact cluster kernel: cells per block
  int cnpx, cnpy, cw, ch;            // cluster kernel: pieces in x and y, the largest piece
  int nbx, nby, nbz;                 // bricks per dimension
  const double* forc;  // Fortran layout (nx+4, ny+4, nz), device
  double* p;           // padded p_non_hydro(:,:,:,taup1), in/out
  double* res;         // padded residual (halo = cyclic copies), updated in place
  double* s[2];        // padded search direction, double-buffered
  double eps;          // congr_epsilon_non_hydro
  int max_it;          // congr_max_itts_non_hydro
  double rtol;         // > 0: extra stop on the recursive residual, sqrt(sum r^2 maskT / sum forc^2 maskT)
  SyncCtl* ctl;
  double* slots;       // 2 * gridDim.x * 4 doubles
  unsigned long long timeout_ns;
  unsigned stall_extra;
  CGResult* out;
};

// Scalar state of congrad_non_hydro's loop (non_hydrostatic.f90:177-242),
// the same in every thread of every block.  The convergence test of
// iteration n needs max|p| of the direction formed after it, so it runs after
// the next iteration's first sweep (after_a).
struct NHCtl {
  enum { kGo = 0, kOk = 1, kErr = 2 };
  double beta = 0, bb = 0, rtol2bb = 0, eps = 0, rtol = 0;
  double betamin = 0, step1 = 0, est = 0, bq = 0, alpha_prev = 0, rr_prev = 0;
  int max_it = 0, n = 0, status = PYOMGPU_OK;

  __device__ int start(double rsold, double bb_, const NHParams& P) {
    beta = rsold;
    bb = bb_;
    rtol = P.rtol;
    rtol2bb = P.rtol * P.rtol * bb;
    eps = P.eps;
    max_it = P.max_it;
    rr_prev = beta;
    if (beta == 0.0) {  // :177
      n = 0;
      return kOk;
    }
    if (max_it < 1) {
      n = 1;
      status = PYOMGPU_MAXITER;
      return kErr;
    }
    n = 1;
    return kGo;
  }
  // after sweep A of iteration n: (s_n, A s_n) and max|s_n| over maskT.  The quotient is formed beside the
  // tests: it is what the next sweep waits for.
  __device__ __forceinline__ int after_a(double sAs, double smax, double& alpha) {
    const double quot = beta / sAs;
    const double step = fabs(alpha_prev) * smax;
    const int m = n - 1;
    if ((m <= 1) | (step < eps) | (est != est) | (rtol > 0.0) | (m >= max_it) | (sAs == 0.0)) {
      if (m >= 1) {  // convergence test of iteration n-1 (:215-226)
        if (m == 1) {
          step1 = step;
          est = step;
          if (step < eps) {
            n = m;
            return kOk;
          }
        } else if (step < eps) {
          const double rate = exp(log(step / step1) / (double)(m - 1));
          est = step * rate / (1.0 - rate);
          if (est < eps) {
            n = m;
            return kOk;
          }
        }
        if (est != est) {
          n = m;
          status = PYOMGPU_NAN;
          return kErr;
        }
        if (rtol > 0.0 && (bb > 0.0 ? rr_prev <= rtol2bb : rr_prev == 0.0)) {
          est = sqrt(rr_prev);
          n = m;
          return kOk;
        }
        if (m >= max_it) {  // :228
          n = max_it + 1;
          status = PYOMGPU_MAXITER;
          return kErr;
        }
      }
      if (sAs == 0.0) return kOk;  // :185
    }
    alpha = quot;
    return kGo;
  }
  // after sweep B of iteration n: rsnew = (res, res) over maskT
  __device__ __forceinline__ int after_b(double rsnew, double alpha) {
    bq = rsnew / beta;  // p = res + rsnew/rsold*p (:189)
    beta = rsnew;
    const double low = fmin(betamin, fabs(rsnew));
    if (n == 1) {  // divergence test (:197-205)
      betamin = fabs(rsnew);
    } else if (n > 2) {
      betamin = low;
      if (fabs(rsnew) > 100.0 * low) {
        status = PYOMGPU_DIVERGED;
        return kErr;
      }
    }
    alpha_prev = alpha;
    rr_prev = rsnew;
    ++n;
    return kGo;
  }
  __device__ void finish(int how, CGResult* out) {
    int converged = 0;
    if (how == kOk) {
      converged = 1;
      status = PYOMGPU_OK;
    } else if (est != est) {
      status = PYOMGPU_NAN;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      out->iterations = n;
      out->converged = converged;
      out->status = status;
      out->est = est;
    }
  }
};

// Arrays of one solve_non_hydrostatic step (non_hydrostatic.f90:5-63), all
// device memory in Fortran layout; the u, v, w, p pointers are already offset
// to their time level.
struct NHStep {
  NHGeo G;
  const double *dxt, *dxu, *dyt, *dyu, *cost, *cosu;  // [nx+4] / [ny+4]
  const double *dzt, *dzw;                            // [nz]
  const uint8_t *maskU, *maskV, *maskW;               // (nx+4, ny+4, nz), 0/1
  double *u, *v, *w;                                  // taup1
  const double *w_tau, *dw_tau, *dw_taum1, *dw_mix;
  double *p1;                                         // p_non_hydro(:,:,:,taup1)
  const double *p0, *pm;                              // tau, taum1
  double* forc;                                       // (nx+4, ny+4, nz) scratch
  double dt_mom, AB_eps;
};
void launch_nh_step_pre(const NHStep& S, cudaStream_t st);
void launch_nh_step_post(const NHStep& S, cudaStream_t st);

const void* nh_cg_kernel_ptr(bool cyclic_x, bool cyclic_y);

// cluster variant for small grids: res, direction and flags distributed over
// the shared memory of up to kNHMaxCluster blocks
constexpr int kNHSmallThreads = 1024;
constexpr int kNHMaxCluster = 16;
constexpr size_t nh_small_smem_bytes(size_t chunk) { return (chunk * 33 + 15) / 16 * 16; }
constexpr size_t kNHSmallSmemMax = 223 * 1024;  // 227 KB per block less room for the static buffers
constexpr int kNHSmallMaxChunk = (int)(kNHSmallSmemMax / 33);
constexpr int kNHSmallMaxCells = kNHMaxCluster * kNHSmallMaxChunk;
constexpr int kNHClusterAuto = 32768;  // automatic choice: the cluster kernel up to this many cells
const void* nh_cg_small_kernel_ptr(bool cyclic_x, bool cyclic_y);

// cluster kernel (nh_clu.cu): pieces of whole columns in the registers and shared memory of one cluster
struct NHCut {
  int npx = 0, npy = 0, w = 0, h = 0, p = 0, nt = 0;
  size_t smem = 0;
  double iter_ns = 0;  // estimated iteration time
};
constexpr int kNHCluNP[][2] = {{128, 4}, {128, 8}, {256, 4}, {256, 8}, {256, 12}};  // threads, levels per thread
// direction with its rim, vertical factors, staged faces, received records (4 words each), reduction slots
__host__ __device__ constexpr size_t nh_clu_smem_bytes(int w, int h, int nz, int p) {
  return 8 * ((size_t)(w + 2) * (h + 2) * ((nz + p - 1) / p * p + 2) + 2 * (size_t)((nz + p - 1) / p * p) +
              4 * (size_t)(w + h) * nz) + 16 + 64 * (size_t)(w + h) * nz + 8 * (size_t)kCluMaxSlots * 16;
}
const void* nh_clu_kernel_ptr(int nt, int p, bool cyclic_x, bool cyclic_y);
void launch_nh_apply(const NHGeo& G, const NHOp& op, const double* p, double* res, cudaStream_t st);
void launch_nh_pack(const NHGeo& G, const double* user, double* padded, cudaStream_t st);
void launch_nh_unpack(const NHGeo& G, const double* padded, double* user, cudaStream_t st);

}  // namespace pyomgpu
