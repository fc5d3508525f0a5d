// lg_trace_common.cuh — small device helpers shared by the trace kernels of both precision
// modes (lg_trace.cu: FP32 scan and double-float solve; lg_exact.cu: exact FP64 solve).
#pragma once
#include "lg_kernels.cuh"

namespace lgd {

__device__ __forceinline__ bool below_cutoff(const float* c, const float* k) {
  return (c[0] < k[0] && c[1] < k[1] && c[2] < k[2]) || c[3] < k[3];
}
__device__ __forceinline__ bool near_cutoff(const float* c, const float* k) {
  bool n = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) n |= fabsf(c[i] - k[i]) <= 1e-6f * k[i];
  return n;
}

// FP32 bounding-circle test shared by both scan passes: false if the object cannot hold a
// hit at a ray parameter <= thr; lb receives a lower bound of its hit distances.
__device__ __forceinline__ bool bound_test(const float4& h, float ox, float oy, float dx, float dy, float thr,
                                           float& lb) {
  const float ocx = h.x - ox, ocy = h.y - oy;
  const float b = ocx * dx + ocy * dy, perp = ocx * dy - ocy * dx;
  const float btol = 2e-6f * (fabsf(b) + fabsf(perp) + h.z) + 1e-6f;
  if (fabsf(perp) > h.z + btol || b + h.z + btol < -TAU32) return false;
  lb = b - h.z - btol;
  return lb <= thr;
}

// The last object of [base, base + n) for which pred holds (0xffffffff: none): the warp's lanes
// try 32 objects at a time, from the end.  Every lane of the warp calls it.
template <class F>
__device__ __forceinline__ uint32_t last_object_of_warp(uint32_t base, uint32_t n, F&& pred) {
  for (uint32_t c = (n + 31) / 32; c-- > 0;) {
    const uint32_t j = c * 32 + lane_id();
    const unsigned hit = __ballot_sync(0xffffffffu, j < n && pred(base + j));
    if (hit) return base + c * 32 + 31u - (unsigned)__clz(hit);
  }
  return 0xffffffffu;
}

// Queued rays a launch takes (the children of the previous generation or step) ...
__device__ __forceinline__ uint64_t n_real_of(const SceneDev& S, const TraceBufs& B, uint32_t gen) {
  if (gen == 0 && !S.serve) return 0;
  const unsigned long long n = B.ctr->queue_count[gen];
  return n < B.queue_cap ? n : B.queue_cap;
}
// ... and primaries it generates (virtual queue entries after the queued ones)
__device__ __forceinline__ uint64_t n_new_of(const SceneDev& S, uint32_t gen) {
  return S.serve ? S.n_new : (gen == 0 ? S.n_primary : 0);
}
__device__ __forceinline__ uint64_t n_in_of(const SceneDev& S, const TraceBufs& B, uint32_t gen) {
  const uint64_t n = n_real_of(S, B, gen) + n_new_of(S, gen);
  return n < B.queue_cap ? n : B.queue_cap;
}

// Time stamps of a generation's kernels (Counters::stamp): the first CTA's start, and for the
// bounce the last CTA's end.  (Event nodes between the kernels of a captured frame cost more than
// the small generations' kernels.)
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ void stamp_start(Counters* ctr, uint32_t gen, int k) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const unsigned long long t = global_ns();
    ctr->stamp[gen][k] = t;
    if (k == 2) atomicMax(&ctr->stamp[gen][3], t);
  }
}
__device__ __forceinline__ void stamp_end(Counters* ctr, uint32_t gen) {
  if (threadIdx.x == 0) atomicMax(&ctr->stamp[gen][3], global_ns());
}

// The threads' event counts into the context's counters, at the end of a kernel: a warp
// reduction (redux) per count, the warps' sums through shared memory, one global atomic per
// CTA and count that is not zero.  Every thread of the CTA calls it.  (A 64-bit atomicAdd on
// shared memory is a compare-and-swap loop: with every thread of the CTA adding to one word,
// the ends of the three trace kernels took most of a small generation: 20 to 34 us a launch
// for 4096 rays, 800 k shared-memory wavefronts.)
template <int N>
__device__ __forceinline__ void add_block_counts(const uint32_t (&v)[N], unsigned long long* const (&dst)[N]) {
  __shared__ unsigned long long part[N][32];
  const unsigned w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int i = 0; i < N; ++i) {  // two halves: the warp's sum may pass 32 bits
    const uint32_t lo = __reduce_add_sync(0xffffffffu, v[i] & 0xffffu), hi = __reduce_add_sync(0xffffffffu, v[i] >> 16);
    if (lane_id() == 0) part[i][w] = ((unsigned long long)hi << 16) + lo;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (threadIdx.x != (unsigned)i) continue;
    unsigned long long sum = 0;
    for (unsigned k = 0; k < nw; ++k) sum += part[i][k];
    if (sum) atomicAdd(dst[i], sum);
  }
}

}  // namespace lgd
