// Weight gradient of a 3x3 convolution (training of the learned
// preconditioner): dW[co][ci][tap] += sum_p G[co][p] X[ci][p + tap - (1,1)],
// db[co] += sum_p G[co][p], bf16 operands, FP32 accumulation.
//
// A contraction over pixels, M = Cin, N = Cout per tap.  In the planar layout
// ([C/8][H][W][8], conv_tc.cuh) eight consecutive pixels of a channel group
// are 8 rows of 16 bytes, which ldmatrix.trans turns into operand fragments at
// any pixel offset, so one staged tile serves all nine taps.  tcgen05 wants
// M = 64 or 128 rows at one stride: with 16 or 32 channels that takes the tap
// shifts as rows, of which at most three in eight (the dx shifts; a row of
// pixels is not a multiple of them) are wanted, and the 16-channel layers at
// full resolution, which dominate, would do 2.7 times the work; so this kernel
// uses warp-level mma.sync, at ~1/4 of the rate but with every product wanted.
//
// A block has nine warps, one per tap; a warp keeps the Cin x Cout block of its
// tap in registers (8 to 64 accumulators; with 64 input channels a block takes
// 32 of the output channels, blockIdx.y) over all tiles the block walks and
// adds it to global memory once at the end.  Tiles of kDwRows x
// kDwCols pixels come by TMA, two stages deep: X with its one-pixel rim
// (zero-filled outside the image), G without.  The maps see a row of pixels as
// 2 W 64-bit elements, so a box row is one contiguous run.  1440x720, all twelve
// layers: 0.59 ms, 4.29 on CUDA cores (one product per shared-memory read).
// Bound, by counters there: the 16-channel layers by the latency of the fragment
// reads and the barrier a tile (LSU pipe a third busy), those of 32 and 64
// channels by the atomic adds at the end, whose queue half of the waits are for.
#include <cuda_bf16.h>

#include <algorithm>

#include "../../include/pyomgpu.h"
#include "common.cuh"
#include "conv_tc.cuh"
#include "tma.cuh"

namespace pyomgpu {

namespace {

constexpr int kDwRows = 4, kDwCols = 64, kDwThreads = 288;
constexpr int kDwBX = kDwCols + 2, kDwBY = kDwRows + 2;

struct DwArgs {
  CUtensorMap map_x, map_g;
  float *dW, *db;
  int tiles_x, ntiles;
  int* err;
  unsigned long long timeout_ns;
};

template <int CIN, int COUT>  // COUT: output channels of a block
struct DwShape {
  static constexpr uint32_t XB = (uint32_t)(CIN / 8) * kDwBY * kDwBX * 16;
  static constexpr uint32_t GB = (uint32_t)(COUT / 8) * kDwRows * kDwCols * 16;
  static constexpr uint32_t GOFF = (XB + 127u) / 128u * 128u;
  static constexpr uint32_t STAGE = (GOFF + GB + 127u) / 128u * 128u;
  static constexpr uint32_t SMEM = 2 * STAGE + 64 + 128;  // + mbarriers + alignment slack
};

__device__ __forceinline__ void ldsm4t(uint32_t a, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kDwThreads) conv_dw_kernel(const __grid_constant__ DwArgs a) {
  using S = DwShape<CIN, COUT>;
  constexpr int MI = CIN / 16, NI = COUT / 16;  // 16 x 16 blocks of the tap's matrix
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
  uint64_t* full = reinterpret_cast<uint64_t*>(base + 2 * S::STAGE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    fence_mbar_init();
  }
  __syncthreads();
  auto issue = [&](int tile, int b) {
    const int ty = tile / a.tiles_x, tx = tile - ty * a.tiles_x;
    uint8_t* s = base + b * S::STAGE;
    mbar_arrive_expect_tx(&full[b], S::XB + S::GB);
    tma_load_3d(s, &a.map_x, 2 * (tx * kDwCols - 1), ty * kDwRows - 1, 0, &full[b]);
    tma_load_3d(s + S::GOFF, &a.map_g, 2 * tx * kDwCols, ty * kDwRows, (int)blockIdx.y * (COUT / 8), &full[b]);
  };
  const int dy = warp / 3, dx = warp - 3 * dy;  // this warp's tap
  // ldmatrix rows: lanes 0-7, 8-15 the two channel groups of pixels 0-7 (A) or the two pixel octets of group 0
  // (B), lanes 16-31 the other eight pixels (A) or the other group (B)
  const int px_a = (lane & 7) + ((lane >> 4) << 3), grp_a = (lane >> 3) & 1;
  const int px_b = (lane & 7) + (((lane >> 3) & 1) << 3), grp_b = lane >> 4;
  const uint32_t off_a = (uint32_t)((grp_a * kDwBY + dy) * kDwBX + dx + px_a) * 16u;
  const uint32_t off_b = S::GOFF + (uint32_t)(grp_b * kDwRows * kDwCols + px_b) * 16u;
  // The matrix unit truncates as it accumulates, so its sums are kept short (the four MMAs of a tile row) and added
  // up in rounded FP32.  With the accumulators in the MMAs over all tiles the gradients of a 1440x720 image were
  // 1e-5 too small where all terms have one sign (6e-8 this way; CUDA-core sums scattered by 2.5e-7).
  float acc[MI][2 * NI][4], accb[2][2] = {};  // accb: warp n has the column sums of G's 16 channels n
#pragma unroll
  for (int n = 0; n < 2 * NI; n++)
#pragma unroll
    for (int m = 0; m < MI; m++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[m][n][e] = 0.f;
  const uint32_t kOne = 0x3f803f80u;  // two bf16 ones
  const uint32_t ones[4] = {kOne, kOne, kOne, kOne};
  bool ok = true;
  int it = 0;
  bool inflight = false;  // the next tile's copies are issued
  if (tid == 0 && (int)blockIdx.x < a.ntiles) issue(blockIdx.x, 0);
  for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, ++it) {
    const int b = it & 1;
    const int next = tile + gridDim.x;
    // the other stage was read to the end before the barrier that closed the previous tile
    if (tid == 0 && next < a.ntiles) {
      fence_proxy_async_smem();
      issue(next, b ^ 1);
    }
    ok = __syncthreads_and(__all_sync(0xffffffffu, mbar_wait_bounded(&full[b], (uint32_t)(it >> 1) & 1u, a.timeout_ns))) != 0;
    inflight = next < a.ntiles;
    if (!ok) break;
    const uint32_t s = smem_u32(base + b * S::STAGE);
#pragma unroll 1
    for (int r = 0; r < kDwRows; r++) {
      float part[MI][2 * NI][4], partb[2][4] = {};  // sums of one tile row
#pragma unroll
      for (int n = 0; n < 2 * NI; n++)
#pragma unroll
        for (int m = 0; m < MI; m++)
#pragma unroll
          for (int e = 0; e < 4; e++) part[m][n][e] = 0.f;
#pragma unroll(CIN * COUT <= 512 ? 4 : 1)
      for (int c = 0; c < kDwCols / 16; c++) {
        const uint32_t pa = s + off_a + (uint32_t)(r * kDwBX + 16 * c) * 16u;
        const uint32_t pb = s + off_b + (uint32_t)(r * kDwCols + 16 * c) * 16u;
        uint32_t fb[NI][4];
#pragma unroll
        for (int n = 0; n < NI; n++) ldsm4t(pb + (uint32_t)(2 * n * kDwRows * kDwCols) * 16u, fb[n]);
#pragma unroll
        for (int m = 0; m < MI; m++) {
          uint32_t fa[4];
          ldsm4t(pa + (uint32_t)(2 * m * kDwBY * kDwBX) * 16u, fa);
#pragma unroll
          for (int n = 0; n < NI; n++) {
            mma16816(part[m][2 * n], fa, fb[n][0], fb[n][1]);
            mma16816(part[m][2 * n + 1], fa, fb[n][2], fb[n][3]);
          }
        }
#pragma unroll
        for (int n = 0; n < NI; n++)
          if (warp == n) {
            mma16816(partb[0], ones, fb[n][0], fb[n][1]);
            mma16816(partb[1], ones, fb[n][2], fb[n][3]);
          }
      }
#pragma unroll
      for (int q = 0; q < 2; q++) {
        accb[q][0] += partb[q][0];
        accb[q][1] += partb[q][1];
      }
#pragma unroll
      for (int n = 0; n < 2 * NI; n++)
#pragma unroll
        for (int m = 0; m < MI; m++)
#pragma unroll
          for (int e = 0; e < 4; e++) acc[m][n][e] += part[m][n][e];
    }
    __syncthreads();
  }
  if (!ok) {
    if (tid == 0) atomicExch(a.err, PYOMGPU_TIMEOUT);
    // let the copies in flight land before the shared memory goes away
    mbar_wait_bounded(&full[it & 1], (uint32_t)(it >> 1) & 1u, a.timeout_ns);
    if (inflight) mbar_wait_bounded(&full[(it + 1) & 1], (uint32_t)((it + 1) >> 1) & 1u, a.timeout_ns);
    return;
  }
  const int co0 = (int)blockIdx.y * COUT;
  // fragment element e of block (m, n): ci = 16 m + lane/4 + 8 (e/2), co = 8 n + 2 (lane%4) + e%2
#pragma unroll
  for (int m = 0; m < MI; m++)
#pragma unroll
    for (int n = 0; n < 2 * NI; n++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int ci = 16 * m + (lane >> 2) + 8 * (e >> 1), co = 8 * n + 2 * (lane & 3) + (e & 1);
        atomicAdd(a.dW + ((size_t)(co0 + co) * CIN + ci) * 9 + warp, acc[m][n][e]);
      }
  if (warp < NI && lane < 4)  // every row of accb holds the sums
#pragma unroll
    for (int q = 0; q < 2; q++) {
      atomicAdd(a.db + co0 + 16 * warp + 8 * q + 2 * lane, accb[q][0]);
      atomicAdd(a.db + co0 + 16 * warp + 8 * q + 2 * lane + 1, accb[q][1]);
    }
}

template <int CIN, int CT>
int launch_one(int cout, const uint16_t* X, const uint16_t* G, int H, int W, float* dW, float* db, int nsm, int* err,
               unsigned long long timeout_ns, cudaStream_t st) {
  using S = DwShape<CIN, CT>;
  static_assert(S::SMEM <= 232448u, "shared memory of one block");
  if (cudaFuncSetAttribute(conv_dw_kernel<CIN, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM) !=
      cudaSuccess)
    return (int)cudaGetLastError();
  DwArgs a{};
  const uint64_t strides[2] = {(uint64_t)W * 16, (uint64_t)W * H * 16};
  const uint64_t dx[3] = {2 * (uint64_t)W, (uint64_t)H, (uint64_t)(CIN / 8)}, dg[3] = {dx[0], dx[1], (uint64_t)(cout / 8)};
  const uint32_t bx[3] = {2 * kDwBX, kDwBY, CIN / 8}, bg[3] = {2 * kDwCols, kDwRows, CT / 8};
  if (encode_map(&a.map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, X, dx, strides, bx) ||
      encode_map(&a.map_g, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, G, dg, strides, bg))
    return -2;
  a.dW = dW;
  a.db = db;
  a.tiles_x = (W + kDwCols - 1) / kDwCols;
  a.ntiles = a.tiles_x * ((H + kDwRows - 1) / kDwRows);
  a.err = err;
  a.timeout_ns = timeout_ns;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, conv_dw_kernel<CIN, CT>, kDwThreads, S::SMEM);
  // more than two blocks an SM would only add more sums at the end
  const int grid = std::max(1, std::min(a.ntiles, std::max(1, std::min(per_sm, 2)) * nsm * CT / cout));
  conv_dw_kernel<CIN, CT><<<dim3(grid, cout / CT), kDwThreads, S::SMEM, st>>>(a);
  return (int)cudaGetLastError();
}

}  // namespace

int conv3x3_dw_launch(int cin, int cout, const uint16_t* X, const uint16_t* G, int H, int W, float* dW, float* db,
                      int nsm, int* err, unsigned long long timeout_ns, cudaStream_t st) {
#define PYOMGPU_DW_CASE(ci, co) \
  if (cin == ci && cout == co) return launch_one<ci, (ci == 64 ? 32 : co)>(co, X, G, H, W, dW, db, nsm, err, timeout_ns, st);
  PYOMGPU_DW_CASE(16, 16)
  PYOMGPU_DW_CASE(16, 32)
  PYOMGPU_DW_CASE(32, 32)
  PYOMGPU_DW_CASE(32, 64)
  PYOMGPU_DW_CASE(64, 64)
  PYOMGPU_DW_CASE(64, 32)
  PYOMGPU_DW_CASE(32, 16)
#undef PYOMGPU_DW_CASE
  return -1;
}

}  // namespace pyomgpu
