// Reductions and halo records inside one thread-block cluster, by tagged words
// (cg_ctl.cuh) pushed into the other blocks' shared memory: the device side of
// the cluster kernels (cg_clu.cu, nh_clu.cu).
#pragma once
#include "cg_clu.cuh"
#include "cg_ctl.cuh"

namespace pyomgpu {
namespace {

__device__ __forceinline__ uint32_t clu_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// cluster shared-memory address of this block's shared address `a` in block `rank`
__device__ __forceinline__ uint32_t clu_map(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// Not the .aligned form: that one is only defined where the whole warp executes it together, and the kernels come
// here from stores that only some lanes make and out of waits that ran out.
__device__ __forceinline__ void clu_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// two tagged words into a block of the cluster, and two of this block's; each
// word is validated on its own, so the pair need not be single-copy atomic
__device__ __forceinline__ void clu_st2(uint32_t a, unsigned long long w0, unsigned long long w1) {
  asm volatile("st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(a), "l"(w0), "l"(w1) : "memory");
}
__device__ __forceinline__ void clu_ld2(uint32_t a, unsigned long long& w0, unsigned long long& w1) {
  asm volatile("ld.relaxed.cluster.shared::cta.v2.u64 {%0, %1}, [%2];" : "=l"(w0), "=l"(w1) : "r"(a) : "memory");
}

// (q, s) as one tagged halo record: 4 words (FP64) or 2 (FP32)
__device__ __forceinline__ void clu_put(uint32_t a, double q, double s, unsigned tag) {
  clu_st2(a, tag_lo(tag, q), tag_hi(tag, q));
  clu_st2(a + 16, tag_lo(tag, s), tag_hi(tag, s));
}
__device__ __forceinline__ void clu_put(uint32_t a, float q, float s, unsigned tag) {
  clu_st2(a, ((unsigned long long)tag << 32) | __float_as_uint(q), ((unsigned long long)tag << 32) | __float_as_uint(s));
}
__device__ __forceinline__ bool clu_get(uint32_t a, double& q, double& s, unsigned tag) {
  unsigned long long w0, w1, w2, w3;
  clu_ld2(a, w0, w1);
  clu_ld2(a + 16, w2, w3);
  q = untag(w0, w1);
  s = untag(w2, w3);
  return tag_ok(w0, tag) && tag_ok(w1, tag) && tag_ok(w2, tag) && tag_ok(w3, tag);
}
__device__ __forceinline__ bool clu_get(uint32_t a, float& q, float& s, unsigned tag) {
  unsigned long long w0, w1;
  clu_ld2(a, w0, w1);
  q = __uint_as_float((unsigned)w0);
  s = __uint_as_float((unsigned)w1);
  return tag_ok(w0, tag) && tag_ok(w1, tag);
}

struct CluRed {
  uint32_t inbox;   // shared address of this block's slots: [parity][pair][value of the pair][kCluMaxSlots] x 16 B
  double* local;    // a block alone in its cluster: [parity][pair][value][warp]
  int nblk, rank;   // blocks in the cluster
  int* err;
  unsigned long long tmo;
};

__device__ __forceinline__ bool clu_expired(int* err, unsigned spin, unsigned long long t0, unsigned long long tmo) {
  if ((spin & 63u) != 0u) return false;
  if (ld_relaxed_i32(err) == 0 && globaltimer_ns() - t0 <= tmo) return false;
  atomicExch(err, PYOMGPU_TIMEOUT);
  return true;
}

// Reduction of (x, y) over all threads of the cluster (kMax: y is a maximum of
// values >= 0), in two halves so that work fits in between.  send: the warp's
// pair goes into the inbox of every block, in the slot of this warp.  recv:
// every warp sums the slots of all warps in one fixed order, so every thread
// has the same bits.  No block barrier: a slot of epoch ep is rewritten at ep+2
// by a warp that has seen every warp's ep+1, i.e. after every warp has read ep.
// `pair` distinguishes the pairs of one epoch.  A block alone in its cluster
// passes the pairs through its own shared memory and one block barrier.
template <int NW, bool kMax>
__device__ __forceinline__ void clu_send(double x, double y, unsigned ep, int pair, const CluRed& R, bool stall) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  x = warp_sum_mma(x);
  y = kMax ? warp_max_nonneg(y) : warp_sum_mma(y);
  const bool upper = lane >= 16;
  const double v = upper ? y : x;
  if (R.nblk == 1 && !stall) {
    if ((lane & 15) == 0) R.local[((((ep & 1u) * 2 + pair) * 2) + (upper ? 1 : 0)) * NW + w] = v;
    return;
  }
  const uint32_t box = R.inbox + (((ep & 1u) * 2 + pair) * 2 + (upper ? 1 : 0)) * (kCluMaxSlots * 16u);
  if ((lane & 15) < R.nblk)
    clu_st2(clu_map(box + 16u * (uint32_t)(R.rank * NW + w), (uint32_t)(lane & 15)), tag_lo(ep, v), tag_hi(ep, v));
}

// False where the wait ran out (the whole warp alike).
template <int NW, bool kMax>
__device__ __forceinline__ bool clu_recv(double& x, double& y, unsigned ep, int pair, const CluRed& R, bool stall) {
  const int lane = threadIdx.x & 31;
  if (R.nblk == 1 && !stall) {
    __syncthreads();
    const double* b = R.local + (((ep & 1u) * 2 + pair) * 2) * NW;
    x = b[0];
    y = b[NW];
#pragma unroll
    for (int k = 1; k < NW; k++) {
      x += b[k];
      y = kMax ? fmax(y, b[NW + k]) : y + b[NW + k];
    }
    return true;
  }
  const int ns = R.nblk * NW;
  const uint32_t box = R.inbox + ((ep & 1u) * 2 + pair) * 2 * (kCluMaxSlots * 16u);
  constexpr int kPer = kCluMaxBlocks * NW / 32;  // slots per lane at most
  double gx[kPer], gy[kPer];
  unsigned long long t0 = 0;
  for (unsigned spin = 0;; spin++) {
    bool ok = true;
#pragma unroll
    for (int m = 0; m < kPer; m++) {
      gx[m] = gy[m] = 0.0;
      int sl = lane + 32 * m;
      if (sl < ns) {
        if (stall && sl == 0) sl = kCluMaxSlots - 1;  // the hook's slot, which nobody writes
        unsigned long long w0, w1, w2, w3;
        clu_ld2(box + 16u * (uint32_t)sl, w0, w1);
        clu_ld2(box + 16u * (uint32_t)(sl + kCluMaxSlots), w2, w3);
        ok = ok && tag_ok(w0, ep) && tag_ok(w1, ep) && tag_ok(w2, ep) && tag_ok(w3, ep);
        gx[m] = untag(w0, w1);
        gy[m] = untag(w2, w3);
      }
    }
    if (__all_sync(0xffffffffu, ok)) break;
    if (spin == 0) t0 = globaltimer_ns();
    if (__any_sync(0xffffffffu, clu_expired(R.err, spin + 1, t0, R.tmo))) return false;
  }
#pragma unroll
  for (int m = 1; m < kPer; m++) {
    gx[0] += gx[m];
    gy[0] = kMax ? fmax(gy[0], gy[m]) : gy[0] + gy[m];
  }
  x = warp_sum_mma(gx[0]);
  y = kMax ? warp_max_nonneg(gy[0]) : warp_sum_mma(gy[0]);
  return true;
}

}  // namespace

}  // namespace pyomgpu
