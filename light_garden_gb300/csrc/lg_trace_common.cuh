// lg_trace_common.cuh — small device helpers shared by the trace kernels of both precision
// modes (lg_trace.cu: FP32 scan and double-float solve; lg_exact.cu: exact FP64 solve).
#pragma once
#include <cstddef>

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

// ------------------------------------------------------------- bulk copy to shared memory
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
  unsigned ok;
  asm volatile(
      "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(d),
      "l"(src), "r"(bytes), "r"(b)
      : "memory");
}

// Stages the ObjScan table into shared memory.  Returns the table to scan: shared memory
// on success, the global table if it does not fit or the bounded wait expired (in which
// case ERR_TMA_TIMEOUT is raised and the caller returns).
static __device__ const ObjScan* stage_objects(const SceneDev& S, ObjScan* sobj, uint64_t* bar, bool fits,
                                        Counters* ctr, bool& failed) {
  failed = false;
  if (!fits || S.n_obj == 0) return S.scan;
  const unsigned bytes = S.n_obj * (unsigned)sizeof(ObjScan);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_expect_tx(bar, bytes);
    const unsigned chunk = 32768u;
    for (unsigned off = 0; off < bytes; off += chunk) {
      const unsigned n = bytes - off < chunk ? bytes - off : chunk;
      bulk_g2s(reinterpret_cast<char*>(sobj) + off, reinterpret_cast<const char*>(S.scan) + off, n, bar);
    }
  }
  __syncthreads();  // barrier initialised before anyone waits on it
  bool done = false;
  const int polls = S.wait_polls;
  for (int it = 0; it < polls && !done; ++it) {
    done = mbar_try_wait(bar, 0);
    if (!done && it > 64) __nanosleep(64);
  }
  if (!done) {
    atomicOr(&ctr->error_flags, ERR_TMA_TIMEOUT);
    // give the copy a last bounded chance to land before this CTA's shared memory is released
    for (int it = 0; it < (1 << 20) && !mbar_try_wait(bar, 0); ++it) __nanosleep(256);
    failed = true;
  }
  __syncthreads();
  return sobj;
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

// Membership of an object at a point known to within delta, decided in FP32 where the FP32 copy
// of its leaves decides it: 1 inside, 0 outside, -1 undecided.  The band of leaf_member32 covers
// delta and the rounding of the point and the leaf parameters to FP32 (1e-6 of the coordinates against
// 6e-8), so a decided answer is the one the precise test gives, outside that test's own band;
// objects the scan only bounds stay undecided.
__device__ __forceinline__ int obj_member32(const ObjScan& s, float px, float py, float delta) {
  if (s.info & INFO_NO_CONTAINS) return 0;
  const uint32_t sk = info_scan(s.info);
  if (sk == SCAN_ONE) {
    const uint32_t ka = info_leaf_a(s.info);
    return ka == LEAF_CUBIC ? -1 : leaf_member32(ka, s.a, px, py, delta);
  }
  if (sk != SCAN_TWO) return -1;
  const int a = leaf_member32(info_leaf_a(s.info), s.a, px, py, delta);
  const int b = leaf_member32(info_leaf_b(s.info), s.b, px, py, delta);
  switch (info_op(s.info)) {
    case LG_OP_AND: return (a == 0 || b == 0) ? 0 : (a == 1 && b == 1 ? 1 : -1);
    case LG_OP_OR: return (a == 1 || b == 1) ? 1 : (a == 0 && b == 0 ? 0 : -1);
    default: return (a == 0 || b == 1) ? 0 : (a == 1 && b == 0 ? 1 : -1);  // a and not b
  }
}

// Queued rays a launch takes (the children of the previous generation or step) ...
__device__ __forceinline__ uint64_t n_real_of(const SceneDev& S, const TraceBufs& B, uint32_t gen) {
  if (gen == 0 && !S.serve) return 0;
  const unsigned long long n = B.ctr->queue_count[gen];
  return n < B.queue_cap ? n : B.queue_cap;
}
// Whether a generation of n queued rays visits them in sorted order: with several scenes always, for
// one from 32768 rays (16384 and 131072 are within 1 % on large frames; the last is late for mixed
// shapes: 64 objects, 32768 primaries 0.98 of the unsorted speed against 1.14).
template <bool MULTI>
__device__ __forceinline__ bool sorts(uint64_t n) {
  return MULTI || n >= 32768;
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

// One queue entry in five 16-byte stores.  (Children built in a local array and copied out went
// through local memory: the exact bounce took 11.1 ms where it takes 7.5, CSG frame at 2^17 rays.)
struct ChildRay {
  uint4 od[2];  // the bits of ox, oy and of dx, dy
  float c[3];
  float ex, ea;
  uint64_t path;
  uint8_t flags, src_leaf;
  uint16_t medium, src_obj;
};
__device__ __forceinline__ void store_child(RayRec* dst, const RayRec& r, const ChildRay& c) {
  static_assert(offsetof(RayRec, path) == 32 && offsetof(RayRec, prim) == 56 && offsetof(RayRec, ex) == 64 &&
                    offsetof(RayRec, medium) == 72 && offsetof(RayRec, src_leaf) == 76 && offsetof(RayRec, scene) == 78,
                "RayRec's layout is spelled out here");
  uint4* u = reinterpret_cast<uint4*>(dst);
  u[0] = c.od[0];
  u[1] = c.od[1];
  u[2] = make_uint4((uint32_t)c.path, (uint32_t)(c.path >> 32), __float_as_uint(c.c[0]), __float_as_uint(c.c[1]));
  u[3] = make_uint4(__float_as_uint(c.c[2]), __float_as_uint(r.c[3]), r.prim,
                    (uint32_t)r.light | ((uint32_t)(uint8_t)(r.gen + 1) << 16) | ((uint32_t)c.flags << 24));
  u[4] = make_uint4(__float_as_uint(c.ex), __float_as_uint(c.ea), (uint32_t)c.medium | ((uint32_t)c.src_obj << 16),
                    (uint32_t)c.src_leaf | ((uint32_t)r.scene << 16));
}

// Places for a warp's segments and children, the reflected rays first, then the refracted ones
// (neighbours of a bundle stay neighbours): one atomic instruction, lane 0 for the ring and lane 1
// for the queue.  All lanes call; each receives its slots.
__device__ __forceinline__ void reserve_out(const TraceBufs& B, uint32_t gen, bool emit, bool child0, bool child1,
                                            unsigned long long& seg, unsigned long long& s0, unsigned long long& s1) {
  const unsigned em = __ballot_sync(0xffffffffu, emit), lane = lane_id();
  const unsigned m0 = __ballot_sync(0xffffffffu, child0), m1 = __ballot_sync(0xffffffffu, child1);
  const unsigned n0 = __popc(m0), need = lane == 0 ? __popc(em) : n0 + __popc(m1);
  unsigned long long at = 0;
  if (lane < 2 && need) at = atomicAdd(lane == 0 ? &B.ctr->seg_count : &B.ctr->queue_count[gen + 1], (unsigned long long)need);
  seg = __shfl_sync(0xffffffffu, at, 0) + __popc(em & lanemask_lt());
  const unsigned long long q0 = __shfl_sync(0xffffffffu, at, 1);
  s0 = q0 + __popc(m0 & lanemask_lt());
  s1 = q0 + n0 + __popc(m1 & lanemask_lt());
}

}  // namespace lgd
