// Cluster-resident Jacobi-PCG (cg_clu.cu): small grids held by the blocks of
// one thread-block cluster.
#pragma once
#include "cg_res.cuh"

namespace pyomgpu {

constexpr int kCluMaxBlocks = 16;  // largest (non-portable) cluster
// Threads per block and points per thread along a column segment (template instances).
constexpr int kCluNT[] = {128, 256};
constexpr int kCluP[] = {4, 6, 8, 12};
// Reduction slots of a block: one per warp of the cluster, and one more for the stall hook.
constexpr int kCluMaxSlots = kCluMaxBlocks * 256 / 32 + 1;

// Field values in shared memory of a piece of at most w x hp points (hp: rows padded to whole column segments)
// with nent boundary entries: direction with its halo, FX, FY, bx, by and the staged boundary values.
__host__ __device__ constexpr size_t clu_fields(int w, int hp, int nent) {
  return (size_t)(w + 2) * (hp + 2) + (size_t)(w + 1) * hp + (size_t)w * (hp + 1) + 2 * (size_t)hp + 2 * (size_t)nent;
}
// Dynamic shared memory of a w x h piece at p points per thread with fields of `es` bytes: the fields, the
// received halo records (4 words of FP64 or 2 of FP32 per entry) and two buffers of two pairs of reduction slots
// (two words per value).
__host__ __device__ constexpr size_t clu_smem_bytes(int w, int h, int p, size_t es) {
  return (es * clu_fields(w, (h + p - 1) / p * p, 2 * (w + h)) + 15) / 16 * 16 + 4 * es * 2 * (size_t)(w + h) +
         8 * (size_t)kCluMaxSlots * 16;
}

// Kernel for nt threads of p points: FP64 fields (surf_press: congrad_surf_press) or FP32 ones.
const void* cg_clu_kernel_ptr(int nt, int p, bool surf_press, bool fp32);

}  // namespace pyomgpu
