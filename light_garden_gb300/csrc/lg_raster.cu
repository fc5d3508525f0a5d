// lg_raster.cu — line accumulation and resolve (sm_103a).
//
// The reference draws its segment list as a 1-px LineList with additive blending into an
// Rgba16Float texture (src/sub_render_pass.rs:43-101, src/light_garden/mod.rs:57-73,
// src/texture_renderer.rs:5) and resolves it with a textured quad
// (src/render_to_texture.wgsl:17-28).  Here:
//   1. k_bin_count / k_scan_tiles / k_build_units / k_bin_scatter sort (segment, tile)
//      pairs into per-tile lists (32 x 32 px tiles) and cut each list into work units;
//   2. k_raster: persistent CTAs take units from a device counter, accumulate the unit's
//      segments into a shared-memory tile with shared atomics (a warp draws a segment, a
//      lane per major-axis pixel), then flush the tile with one global atomic per pixel
//      channel.  Fixed-point (int64 Q31.32) sums make the image independent of the order
//      in which units and segments are processed, so it is bit-reproducible;
//   3. k_resolve_f16: Q31.32 -> f32 -> binary16 (RNE), 8 B per pixel.
#include <cuda_fp16.h>

#include <type_traits>

#include "lg_kernels.cuh"
#include "lg_trace_common.cuh"

namespace lgd {

// ------------------------------------------------------------------ blend helpers
__device__ __forceinline__ float blend_factor(int f, int ch, const float* src, const float* k) {
  switch (f) {
    case LG_BF_ZERO: return 0.0f;
    case LG_BF_ONE: return 1.0f;
    case LG_BF_SRC: return src[ch];
    case LG_BF_ONE_MINUS_SRC: return __fsub_rn(1.0f, src[ch]);
    case LG_BF_SRC_ALPHA: return src[3];
    case LG_BF_ONE_MINUS_SRC_ALPHA: return __fsub_rn(1.0f, src[3]);
    case LG_BF_CONSTANT: return k[ch];
    default: return __fsub_rn(1.0f, k[ch]);
  }
}

__device__ __forceinline__ float contribution(const BlendDev& B, int ch, const float* src) {
  if (B.op[ch] == LG_BO_MIN || B.op[ch] == LG_BO_MAX) return src[ch];
  return __fmul_rn(src[ch], blend_factor(B.src[ch], ch, src, B.constant));
}

__device__ __forceinline__ long long ident64(int op) {
  return op == LG_BO_MIN ? 0x7fffffffffffffffll : (op == LG_BO_MAX ? (long long)0x8000000000000000ull : 0ll);
}
__device__ __forceinline__ float ident32(int op) {
  return op == LG_BO_MIN ? INFINITY : (op == LG_BO_MAX ? -INFINITY : 0.0f);
}

// ------------------------------------------------------------------ clear
template <class V4, class V>
__device__ __forceinline__ void fill_px(void* img, uint64_t n, V r, V g, V b, V a) {
  V4 c;
  c.x = r; c.y = g; c.z = b; c.w = a;
  V4* p = reinterpret_cast<V4*>(img);
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = c;
}
__global__ void k_clear_accum(RasterArgs A) {
  const uint64_t n = (uint64_t)A.W * A.H;
  const float* c = A.blend.clear;
  if (A.acc == ACC_I64)
    fill_px<longlong4_32a, long long>(A.accum, n, to_fixed(c[0]), to_fixed(c[1]), to_fixed(c[2]), to_fixed(c[3]));
  else if (A.acc == ACC_F64)
    fill_px<double4_32a, double>(A.accum, n, c[0], c[1], c[2], c[3]);
  else
    fill_px<float4, float>(A.accum, n, c[0], c[1], c[2], c[3]);
}

__global__ void k_accum_f32(const double* src, float* dst, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = __double2float_rn(src[i]);
}

// adds a term to value k of an FP64 or FP32 accumulation image
__device__ __forceinline__ void image_add(const RasterArgs& A, uint64_t k, double v) {
  if (A.acc == ACC_F64) atomicAdd(reinterpret_cast<double*>(A.accum) + k, v);
  else atomicAdd(reinterpret_cast<float*>(A.accum) + k, __double2float_rn(v));
}

// ------------------------------------------------------------------ canvases
// The canvas a segment or a bin belongs to: the context's one canvas, or in a
// multi-scene accumulation the scene's own.
struct CanvasLoc {
  uint32_t W, H, ntx;
  uint64_t bin_base, px_base;
};
__device__ __forceinline__ CanvasLoc canvas_one(const RasterArgs& A) {
  CanvasLoc C;
  C.W = A.W; C.H = A.H; C.ntx = A.ntx; C.bin_base = 0; C.px_base = 0;
  return C;
}
__device__ __forceinline__ CanvasLoc canvas_at(const RasterArgs& A, uint32_t s) {
  const SceneCanvas& K = A.canvases[s];
  CanvasLoc C;
  C.W = K.W; C.H = K.H; C.ntx = K.ntx; C.bin_base = K.bin_base; C.px_base = K.px_base;
  return C;
}
__device__ __forceinline__ CanvasLoc canvas_of_bin(const RasterArgs& A, uint64_t bin) {
  if (!A.seg_scene) return canvas_one(A);
  uint32_t lo = 0, hi = A.n_scenes;  // the last scene whose first bin is <= bin
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (A.canvases[mid].bin_base <= bin) lo = mid; else hi = mid;
  }
  return canvas_at(A, lo);
}

// ------------------------------------------------------------------ binning
// The tiles that tile column tm (major-axis tiles) of a segment touches: the minor range is
// bounded by the samples at the column's two ends, since v(i) is monotone in i, and with
// |slope| <= 1 it spans at most two tiles.
template <class F>
__device__ __forceinline__ void column_tiles(const RSetup& R, const CanvasLoc& A, int tm, F&& f) {
  const int nmin = (int)(R.xmajor ? A.H : A.W);
  const int a = max(R.lo, tm * TILE), b = min(R.hi, tm * TILE + TILE) - 1;
  const int ja = raster_minor(R, a), jb = raster_minor(R, b);
  int jlo = min(ja, jb), jhi = max(ja, jb);
  if (jhi < 0 || jlo >= nmin) return;
  jlo = max(jlo, 0);
  jhi = min(jhi, nmin - 1);
  for (int tn = jlo / TILE; tn <= jhi / TILE; ++tn) {
    // bin id = 2 * tile + orientation: x-major and y-major segments of a tile are
    // rasterised in separate units, each with a bank-conflict-free layout
    const uint32_t tile = R.xmajor ? (uint32_t)tn * A.ntx + (uint32_t)tm : (uint32_t)tm * A.ntx + (uint32_t)tn;
    f((uint32_t)(A.bin_base + 2u * tile + (R.xmajor ? 0u : 1u)));
  }
}

// Visits every tile that holds at least one pixel of the segment.
template <class F>
__device__ __forceinline__ void for_each_tile(const RSetup& R, const CanvasLoc& A, F&& f) {
  const int tlo = R.lo / TILE, thi = (R.hi - 1) / TILE;
  for (int tm = tlo; tm <= thi; ++tm) column_tiles(R, A, tm, f);
}

__device__ __forceinline__ uint64_t n_segments(const RasterArgs& A) {
  const unsigned long long n = A.ctr->seg_count;
  return n < A.seg_cap ? n : A.seg_cap;
}

// Every (segment, bin) pair of the calling warp's share of the segments (32 consecutive
// segments per warp step, warp-strided over the grid), with the lanes spread densely over
// the step's tile columns: the 32 segments are set up lane-parallel, their column counts
// prefix-summed, and lane L takes columns L, L + 32, ... of the step, finding each column's
// segment by a binary search over the prefix sums with shuffles.  A segment that crosses
// many tiles is shared by the warp instead of keeping 31 lanes waiting.  f(segment, bin).
// Every lane of the warp calls it (the loops are warp-uniform).  own(segment) is called once for
// every segment that has columns on its canvas.
struct NoOwn {
  __device__ __forceinline__ void operator()(uint64_t) const {}
};
template <class F, class G = NoOwn>
__device__ __forceinline__ void for_each_pair_dense(const RasterArgs& A, uint64_t n, F&& f, G&& own = G()) {
  const unsigned lane = lane_id();
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t base = ((blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5) * 32; base < n; base += nw * 32) {
    const uint64_t i = base + lane;
    RSetup R;
    R.xmajor = 0; R.ua = 0.0f; R.va = 0.0f; R.slope = 0.0f; R.lo = 0; R.hi = 0;
    uint32_t sc = 0;
    int cnt = 0;
    if (i < n) {
      const float4 g = __ldg(reinterpret_cast<const float4*>(A.segs + i));
      if (A.seg_scene) sc = A.seg_scene[i];
      const CanvasLoc C = A.seg_scene ? canvas_at(A, sc) : canvas_one(A);
      lg_segment sg;
      sg.x0 = g.x; sg.y0 = g.y; sg.x1 = g.z; sg.y1 = g.w;
      if (raster_setup(sg, C.W, C.H, R)) {
        cnt = (R.hi - 1) / TILE - R.lo / TILE + 1;
        own(i);
      }
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)lane >= o) incl += y;
    }
    const int excl = incl - cnt;
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    for (int p0 = 0; p0 < total; p0 += 32) {
      const int p = p0 + (int)lane;
      // owner: the last lane whose exclusive prefix is <= p (a lane without columns shares
      // its prefix with the next lane and loses the search to it)
      int k = 0;
#pragma unroll
      for (int st = 16; st > 0; st >>= 1)
        if (__shfl_sync(0xffffffffu, excl, k + st) <= p) k += st;
      RSetup Q;
      Q.xmajor = __shfl_sync(0xffffffffu, R.xmajor, k);
      Q.ua = __shfl_sync(0xffffffffu, R.ua, k);
      Q.va = __shfl_sync(0xffffffffu, R.va, k);
      Q.slope = __shfl_sync(0xffffffffu, R.slope, k);
      Q.lo = __shfl_sync(0xffffffffu, R.lo, k);
      Q.hi = __shfl_sync(0xffffffffu, R.hi, k);
      const uint32_t qsc = __shfl_sync(0xffffffffu, sc, k);
      const int qexcl = __shfl_sync(0xffffffffu, excl, k);
      if (p < total) {
        const CanvasLoc C = A.seg_scene ? canvas_at(A, qsc) : canvas_one(A);
        const uint64_t seg = base + (uint64_t)k;
        column_tiles(Q, C, Q.lo / TILE + (p - qexcl), [&](uint32_t bin) { f(seg, bin); });
      }
    }
  }
}

// Per-CTA tile histogram in shared memory (native 32-bit shared atomics), one global
// atomic per touched tile per CTA.  Falls back to warp-aggregated global atomics when the
// tile count does not fit (smem_tiles == 0).
__global__ void __launch_bounds__(SCATTER_THREADS) k_bin_count(RasterArgs A, int smem_tiles) {
  if (A.ctr->skip_raster) return;
  extern __shared__ unsigned hist[];
  __shared__ unsigned cta_max[4];
  const uint64_t n = n_segments(A);
  if (threadIdx.x < 4) cta_max[threadIdx.x] = 0u;
  if (smem_tiles)
    for (uint32_t t = threadIdx.x; t < A.n_tiles; t += blockDim.x) hist[t] = 0;
  __syncthreads();
  uint32_t my_refs = 0;
  unsigned my_max[4] = {0u, 0u, 0u, 0u};
  auto color_max = [&](uint64_t i) {  // the colour shares the coordinates' sector
    if (!A.scaled) return;
    const uint4 c = __ldg(reinterpret_cast<const uint4*>(A.segs + i) + 1);
    const unsigned m[4] = {c.x & 0x7fffffffu, c.y & 0x7fffffffu, c.z & 0x7fffffffu, c.w & 0x7fffffffu};
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) my_max[ch] = max(my_max[ch], m[ch] < 0x7f800000u ? m[ch] : 0u);
  };
  for_each_pair_dense(A, n, [&](uint64_t, uint32_t tile) {
    ++my_refs;
    if (smem_tiles) {
      atomicAdd(&hist[tile], 1u);
    } else {
      const unsigned act = __activemask();
      const unsigned grp = __match_any_sync(act, tile);
      const int leader = __ffs(grp) - 1;
      if ((int)lane_id() == leader) atomicAdd(&A.tile_count[tile], (unsigned)__popc(grp));
    }
  }, color_max);
  if (A.scaled) {
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
      const unsigned m = __reduce_max_sync(0xffffffffu, my_max[ch]);
      if (lane_id() == 0 && m) atomicMax(&cta_max[ch], m);
    }
    __syncthreads();
    if (threadIdx.x < 4 && cta_max[threadIdx.x]) atomicMax(&A.ctr->color_max[threadIdx.x], cta_max[threadIdx.x]);
  }
  if (smem_tiles) {
    __syncthreads();
    uint32_t* mine = A.cta_hist ? A.cta_hist + (uint64_t)blockIdx.x * A.n_tiles : nullptr;
    for (uint32_t t = threadIdx.x; t < A.n_tiles; t += blockDim.x) {
      const unsigned c = hist[t];
      if (mine) mine[t] = c;
      if (c) atomicAdd(&A.tile_count[t], c);
    }
  }
  add_block_counts<1>({my_refs}, {&A.ctr->bin_refs});
}

// Segments per raster unit of this accumulation.  A unit ends with the flush of its 32 KB tile,
// so big accumulations take the largest units the sums allow; a small one is cut finer, down
// to one round of the CTA's eight warps, until every CTA has about three units: a tile that
// holds a light source has as many segments as the light has rays, and as one unit it kept a
// single CTA busy for most of a small frame (334 us of raster in a frame of 12,000 rays).
__device__ __forceinline__ uint32_t unit_refs_of(const RasterArgs& A) {
  const unsigned long long share = A.ctr->bin_refs / max(A.unit_share, 1u);
  const unsigned long long u = (share + MIN_UNIT_REFS - 1) / MIN_UNIT_REFS * MIN_UNIT_REFS;
  return (uint32_t)(u < MIN_UNIT_REFS ? MIN_UNIT_REFS : u > A.unit_refs ? A.unit_refs : u);
}

// single-CTA exclusive scan of refs and units per tile
__global__ void __launch_bounds__(1024) k_scan_tiles(RasterArgs A) {
  if (A.ctr->skip_raster) return;
  __shared__ unsigned long long wsum_r[32], wsum_u[32];
  __shared__ unsigned long long carry_r, carry_u;
  if (threadIdx.x == 0) { carry_r = 0; carry_u = 0; }
  __syncthreads();
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const uint32_t per = unit_refs_of(A);
  for (uint32_t base = 0; base < A.n_tiles; base += blockDim.x) {
    const uint32_t t = base + threadIdx.x;
    const uint32_t cn = t < A.n_tiles ? A.tile_count[t] : 0u;
    const unsigned long long c = cn, u = ((unsigned long long)cn + per - 1) / per;
    unsigned long long ir = c, iu = u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long yr = __shfl_up_sync(0xffffffffu, ir, o), yu = __shfl_up_sync(0xffffffffu, iu, o);
      if ((int)lane >= o) { ir += yr; iu += yu; }
    }
    if (lane == 31) { wsum_r[wid] = ir; wsum_u[wid] = iu; }
    __syncthreads();
    if (wid == 0) {
      unsigned long long sr = lane < (blockDim.x >> 5) ? wsum_r[lane] : 0ull;
      unsigned long long su = lane < (blockDim.x >> 5) ? wsum_u[lane] : 0ull;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long yr = __shfl_up_sync(0xffffffffu, sr, o), yu = __shfl_up_sync(0xffffffffu, su, o);
        if ((int)lane >= o) { sr += yr; su += yu; }
      }
      wsum_r[lane] = sr;
      wsum_u[lane] = su;
    }
    __syncthreads();
    const unsigned long long pr = (wid ? wsum_r[wid - 1] : 0ull) + ir - c + carry_r;
    const unsigned long long pu = (wid ? wsum_u[wid - 1] : 0ull) + iu - u + carry_u;
    if (t < A.n_tiles) {
      A.tile_off[t] = pr;
      A.tile_cursor[t] = pr;
      A.unit_off[t] = pu;
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) {
      carry_r = pr + c;
      carry_u = pu + u;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    A.ctr->tile_refs = carry_r;
    A.ctr->units = carry_u;
    A.ctr->unit_cursor = 0;
  }
}

// Multi-block version of k_scan_tiles for the many bins of a multi-scene accumulation:
// per-CTA sums of refs and units, one scan of the CTA sums, then each CTA scans its own
// chunk from its offset.  part holds 2 values per CTA (refs, units).
__device__ __forceinline__ void tile_counts(const RasterArgs& A, uint32_t per, uint32_t t, unsigned long long& c,
                                            unsigned long long& u) {
  c = t < A.n_tiles ? A.tile_count[t] : 0ull;
  u = (c + per - 1) / per;
}

// inclusive block scan of (r, u) over 1024 threads; returns the block totals in tr, tu
__device__ __forceinline__ void block_scan2(unsigned long long& r, unsigned long long& u, unsigned long long& tr,
                                            unsigned long long& tu) {
  __shared__ unsigned long long wr[32], wu[32];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long yr = __shfl_up_sync(0xffffffffu, r, o), yu = __shfl_up_sync(0xffffffffu, u, o);
    if ((int)lane >= o) { r += yr; u += yu; }
  }
  if (lane == 31) { wr[wid] = r; wu[wid] = u; }
  __syncthreads();
  if (wid == 0) {
    unsigned long long sr = lane < (blockDim.x >> 5) ? wr[lane] : 0ull;
    unsigned long long su = lane < (blockDim.x >> 5) ? wu[lane] : 0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long yr = __shfl_up_sync(0xffffffffu, sr, o), yu = __shfl_up_sync(0xffffffffu, su, o);
      if ((int)lane >= o) { sr += yr; su += yu; }
    }
    wr[lane] = sr;
    wu[lane] = su;
  }
  __syncthreads();
  if (wid) { r += wr[wid - 1]; u += wu[wid - 1]; }
  tr = wr[(blockDim.x >> 5) - 1];
  tu = wu[(blockDim.x >> 5) - 1];
  __syncthreads();
}

__global__ void __launch_bounds__(1024) k_tiles_partial(RasterArgs A, unsigned long long* part) {
  if (A.ctr->skip_raster) return;
  const uint32_t b0 = blockIdx.x * (uint32_t)TILE_SCAN_CHUNK, per = unit_refs_of(A);
  unsigned long long r = 0, u = 0;
  for (uint32_t k = threadIdx.x; k < (uint32_t)TILE_SCAN_CHUNK; k += blockDim.x) {
    unsigned long long c, v;
    tile_counts(A, per, b0 + k, c, v);
    r += c;
    u += v;
  }
  unsigned long long tr, tu;
  block_scan2(r, u, tr, tu);
  if (threadIdx.x == 0) { part[2 * blockIdx.x] = tr; part[2 * blockIdx.x + 1] = tu; }
}

__global__ void __launch_bounds__(1024) k_tiles_scan_partials(RasterArgs A, unsigned long long* part, uint32_t n_part) {
  if (A.ctr->skip_raster) return;
  __shared__ unsigned long long carry_r, carry_u;
  if (threadIdx.x == 0) { carry_r = 0; carry_u = 0; }
  __syncthreads();
  for (uint32_t base = 0; base < n_part; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const unsigned long long c = i < n_part ? part[2 * i] : 0ull, v = i < n_part ? part[2 * i + 1] : 0ull;
    unsigned long long r = c, u = v, tr, tu;
    block_scan2(r, u, tr, tu);
    const unsigned long long cr = carry_r, cu = carry_u;
    if (i < n_part) { part[2 * i] = cr + r - c; part[2 * i + 1] = cu + u - v; }
    __syncthreads();
    if (threadIdx.x == 0) { carry_r = cr + tr; carry_u = cu + tu; }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    A.ctr->tile_refs = carry_r;
    A.ctr->units = carry_u;
    A.ctr->unit_cursor = 0;
  }
}

__global__ void __launch_bounds__(1024) k_tiles_apply(RasterArgs A, const unsigned long long* part) {
  if (A.ctr->skip_raster) return;
  __shared__ unsigned long long carry_r, carry_u;
  if (threadIdx.x == 0) { carry_r = part[2 * blockIdx.x]; carry_u = part[2 * blockIdx.x + 1]; }
  __syncthreads();
  const uint32_t b0 = blockIdx.x * (uint32_t)TILE_SCAN_CHUNK, per = unit_refs_of(A);
  for (uint32_t k = 0; k < (uint32_t)TILE_SCAN_CHUNK; k += blockDim.x) {
    const uint32_t t = b0 + k + threadIdx.x;
    unsigned long long c, v;
    tile_counts(A, per, t, c, v);
    unsigned long long r = c, u = v, tr, tu;
    block_scan2(r, u, tr, tu);
    const unsigned long long cr = carry_r, cu = carry_u;
    if (t < A.n_tiles) {
      A.tile_off[t] = cr + r - c;
      A.tile_cursor[t] = cr + r - c;
      A.unit_off[t] = cu + u - v;
    }
    __syncthreads();
    if (threadIdx.x == 0) { carry_r = cr + tr; carry_u = cu + tu; }
    __syncthreads();
  }
}

// After each generation of a streaming accumulation: accumulate now only if the ring could
// not take the next generation (one segment per queued ray at most), or nothing follows.
__global__ void k_stream_decide(Counters* ctr, uint32_t gen, uint64_t seg_cap, uint64_t queue_cap, int last) {
  const unsigned long long next = ctr->queue_count[gen + 1];
  const unsigned long long nxt = next < queue_cap ? next : queue_cap;
  const bool go = last || next == 0 || ctr->seg_count + nxt > seg_cap;
  ctr->skip_raster = go ? 0u : 1u;
}

__global__ void k_clear_counts(RasterArgs A) {
  if (A.ctr->skip_raster) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.ctr->bin_refs = 0;
    for (int ch = 0; ch < 4; ++ch) A.ctr->color_max[ch] = 0u;
  }
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < A.n_tiles; t += gridDim.x * blockDim.x) A.tile_count[t] = 0u;
}

// End of one generation of a streaming accumulation: totals, largest demands, and the
// segment ring emptied for the next generation.
__global__ void k_stream_rotate(Counters* ctr, uint64_t seg_cap) {
  if (ctr->skip_raster) return;
  const unsigned long long s = ctr->seg_count, r = ctr->tile_refs;
  ctr->seg_total += s < seg_cap ? s : seg_cap;
  if (s > ctr->seg_max) ctr->seg_max = s;
  ctr->refs_total += r;
  if (r > ctr->refs_max) ctr->refs_max = r;
  ctr->seg_count = 0;
}

__global__ void k_build_units(RasterArgs A) {
  if (A.ctr->skip_raster) return;
  const uint32_t per = unit_refs_of(A);
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < A.n_tiles; t += gridDim.x * blockDim.x) {
    const uint64_t c = A.tile_count[t], off = A.tile_off[t];
    uint64_t u = A.unit_off[t];
    for (uint64_t b = 0; b < c; b += per, ++u) {
      if (u >= A.units_cap) return;
      Unit U;
      U.tile = t;
      U.begin = off + b;
      U.n = (uint32_t)(c - b < per ? c - b : per);
      A.units[u] = U;
    }
  }
}

// Scatter of segment ids into the per-tile lists.  With shared-memory tiles a CTA counts
// its own segments per tile, reserves one range per touched tile with a single global
// atomic, and fills the ranges through shared-memory cursors.
__global__ void __launch_bounds__(SCATTER_THREADS) k_bin_scatter(RasterArgs A, int smem_tiles) {
  if (A.ctr->skip_raster) return;
  extern __shared__ unsigned cur[];  // slots are < refs_cap < 2^32
  const uint64_t n = n_segments(A);
  if (smem_tiles) {
    if (A.cta_hist) {  // this CTA's counts, left by k_bin_count with the same launch shape
      const uint32_t* mine = A.cta_hist + (uint64_t)blockIdx.x * A.n_tiles;
      for (uint32_t t = threadIdx.x; t < A.n_tiles; t += blockDim.x) cur[t] = mine[t];
    } else {
      for (uint32_t t = threadIdx.x; t < A.n_tiles; t += blockDim.x) cur[t] = 0;
      __syncthreads();
      for_each_pair_dense(A, n, [&](uint64_t, uint32_t tile) { atomicAdd(&cur[tile], 1u); });
    }
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < A.n_tiles; t += blockDim.x) {
      const unsigned c = cur[t];
      cur[t] = c ? (unsigned)atomicAdd(&A.tile_cursor[t], (unsigned long long)c) : 0u;
    }
    __syncthreads();
    for_each_pair_dense(A, n, [&](uint64_t i, uint32_t tile) {
      const unsigned slot = atomicAdd(&cur[tile], 1u);
      if (slot < A.refs_cap) A.refs[slot] = (uint32_t)i;
    });
    return;
  }
  for_each_pair_dense(A, n, [&](uint64_t i, uint32_t tile) {
    const unsigned act = __activemask();
    const unsigned grp = __match_any_sync(act, tile);
    const int leader = __ffs(grp) - 1;
    unsigned long long base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(&A.tile_cursor[tile], (unsigned long long)__popc(grp));
    base = __shfl_sync(grp, base, leader);
    const unsigned long long slot = base + __popc(grp & lanemask_lt());
    if (slot < A.refs_cap) A.refs[slot] = (uint32_t)i;
  });
}

// ------------------------------------------------------------------ tile raster
constexpr int TILE_PX = TILE * TILE;  // cells of a tile
// Words between two sum planes: the flush reads the four channels of eight cells per warp, and
// two planes (one channel) are 8 banks apart, so its 32 reads fall in 32 banks.
constexpr int PLANE = TILE_PX + 4;

// Layout of a unit's shared-memory tile: x-major units index cells [row][col] and their
// 32 lanes own 32 columns; y-major units index [col][row] and their lanes own 32 rows.
// Either way one warp's 32 accesses fall in 32 distinct banks.
//
// Additive sums are exact split sums in native 32-bit shared atomics: a term of magnitude
// below 2^(LIMIT - FRAC) is a whole number |q| < 2^LIMIT of units 2^-FRAC, split as
// |q| = b * 2^SPLIT + c, and a negative term negates both.  A unit holds at most UNIT_MAX
// segments and a segment adds at most once to a pixel, so both plane sums stay within 32
// signed bits and B * 2^SPLIT + C is exact.
//   FIXED: Q31.32, q rounded to nearest even (to_fixed); terms of 4 and more take 64-bit
//     atomics on the image instead, which is just as exact.
//   F32: units of 2^(E - 42), where 2^E is a power of two above the channel's terms (term_exponent);
//     every FP32 value in [2^(E - 19), 2^E) is whole in them, so a unit's sum is the exact sum of its
//     terms, and the FP64 image (accum_kind) adds the units.  A unit with smaller terms is drawn again
//     for the next windows of 19 exponents, F32_PASSES windows in all, with only the segments that have
//     terms there.  What is left (NaN, infinities, terms above 2^64 or below the windows) takes atomics
//     on the image.  Fixed units of 2^-41, with atomics for every term outside [2^-18, 2), took
//     20.1 ms for a 64-object frame of lights of (1, 0.002, 0), where this takes 4.5; 63.4 ms for lights
//     of alpha 0.0015 beside control lines of alpha 1, now 8.1; and 1.53 ms for 400 k segments with a
//     channel near 1e-6, now 0.23.  Unit colours: 3.95 and 4.00 ms, 0.221 and 0.228 ms.
enum RasterMode { RM_FIXED_SPLIT = 0, RM_FIXED_MINMAX = 1, RM_F32 = 2, RM_F32_MINMAX = 3 };
constexpr int F32_PASSES = 3, F32_WINDOW = 19;
template <int MODE>
struct Split {
  static constexpr bool on = MODE == RM_FIXED_SPLIT || MODE == RM_F32;
  static constexpr int frac = 32;  // FIXED
  static constexpr int bits = MODE == RM_F32 ? 21 : 17;   // c = |q| mod 2^bits
  static constexpr int limit = MODE == RM_F32 ? 42 : 34;  // |q| < 2^limit
  static constexpr uint32_t unit_max = MODE == RM_F32 ? F32_UNIT_REFS : SPLIT_UNIT_REFS;
  static_assert((1ll << (limit - bits)) * unit_max <= (1ll << 31) && (1ll << bits) * unit_max <= (1ll << 31),
                "split plane sums must fit 32 bits");
};

template <int MODE>
struct RasterSmem {
  static constexpr int acc_words = MODE == RM_F32_MINMAX ? 4 * TILE_PX : MODE == RM_FIXED_MINMAX ? 8 * TILE_PX : 8 * PLANE;
  static constexpr int stage_words = 8 * 32 * 12;  // 8 warps x 32 staged segments x 48 B
  static constexpr int owner_words = 8 * 32 * 32 / 4;  // 8 warps x 1024 (segment, column) pairs, 1 B each
  static constexpr int pref_words = 8 * 33;
  static constexpr int bytes = (acc_words + stage_words + owner_words + pref_words) * 4;
};

// one staged segment: raster setup restricted to the unit's tile and the per-channel
// source terms, 48 B
struct __align__(16) Staged {
  float ua, va, slope;
  unsigned mask;        // the tile's major-axis pixels it covers (one run of bits)
  unsigned q[8];        // split sums: (c, b) per channel; FIXED_MINMAX: 4 x int64; F32_MINMAX: 4 x float
};

// |q| = b * 2^bits + c of a term whose magnitude is t < 2^bits in units of 2^bits (a power of two
// times the term: exact); n: negative.  The fraction of t and its scaling are exact, so rounding
// the fraction rounds t * 2^bits (the carry of a rounded-up fraction goes to b).  The FP32 steps
// take the place of a 64-bit float conversion, which issues on the FP64 pipe.
template <int MODE>
__device__ __forceinline__ void split_bits(float t, bool n, unsigned& c_out, unsigned& b_out) {
  using S = Split<MODE>;
  const float f = floorf(t);
  int b = (int)f, c = __float2int_rn((t - f) * (float)(1 << S::bits));
  if (MODE == RM_FIXED_SPLIT && c == (1 << S::bits)) {
    c = 0;
    ++b;
  }
  c_out = (unsigned)(n ? -c : c);
  b_out = (unsigned)(n ? -b : b);
}

// A fixed-point term's split; false when it is out of the split's range.
__device__ __forceinline__ bool split_fixed(float v, bool neg, unsigned& c_out, unsigned& b_out) {
  using S = Split<RM_FIXED_SPLIT>;
  if (v != v) v = 0.0f;  // to_fixed: NaN adds nothing
  const float m = fabsf(v);
  if (!(m < (float)(1ll << (S::limit - S::frac)))) return false;
  split_bits<RM_FIXED_SPLIT>(m * (float)(1 << (S::frac - S::bits)), (v < 0.0f) != neg, c_out, b_out);
  return true;
}

// F32: E of a channel (see Split): a power of two above its terms' magnitudes, from those of the
// colours and the blend factor, within the range in which all scales are normal FP32 numbers.
__device__ __forceinline__ int term_exponent(const RasterArgs& A, int ch) {
  auto above = [](unsigned bits) { return (int)(bits >> 23) - 126; };
  const int c = above(A.ctr->color_max[ch]), a = above(A.ctr->color_max[3]);
  const float k = A.blend.constant[ch];
  int f = 0;
  switch (A.blend.src[ch]) {
    case LG_BF_SRC: f = c; break;
    case LG_BF_ONE_MINUS_SRC: f = max(c, 0) + 1; break;
    case LG_BF_SRC_ALPHA: f = a; break;
    case LG_BF_ONE_MINUS_SRC_ALPHA: f = max(a, 0) + 1; break;
    case LG_BF_CONSTANT: f = above(__float_as_uint(fabsf(k))); break;
    case LG_BF_ONE_MINUS_CONSTANT: f = above(__float_as_uint(fabsf(1.0f - k))); break;
    default: break;
  }
  return min(max(c + f, -60), 64);
}
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }

__device__ __forceinline__ void shared_add(unsigned addr, unsigned v) {
  asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ void f32_minmax(float* p, float v, bool mn) {
  float o = *p;
  while (mn ? v < o : v > o) {
    const float w = __int_as_float(atomicCAS(reinterpret_cast<int*>(p), __float_as_int(o), __float_as_int(v)));
    if (w == o) break;
    o = w;
  }
}

// A batch of 32 segments is drawn segment by segment, a lane per column of the tile, when its
// segments cover at least this many columns each on average; else its (segment, column) pairs
// are spread densely over the lanes.  Drawing by segments reads its parameters from shared
// memory once per warp (a broadcast) and its atomics hit 32 banks; the dense walk takes about three
// times the instructions for 32 pairs and its lanes' rows collide.  (400 k segments of 12 px: 171 us
// a call with 12 here, 178 with 8 or 5; of 90 px: 253, 253, 257.)
#ifndef LG_RASTER_LANE_MIN
#define LG_RASTER_LANE_MIN 12
#endif

// Bound: the shared-memory pipe.  A segment takes seven or eight 32-bit atomics per tile and two
// or three 16-byte broadcast reads, two wavefronts each: 94 % of the L1 wavefront slots on the mid
// scene at 2^15 rays per light with three reads; two reads take 2.40 ms where three take 2.65 (mid
// scene, 2^14 rays per light) and 10.6 where 11.4 (CSG frame, 2^17 rays).  Spreading every pixel over
// the lanes, with a branch per atomic, took 2.78 ms at 2^13 rays per light; masked terms, a lane
// per column, 1.42 ms (2196 M against 1030 M warp instructions, 167 M against 10 M bank conflicts).
template <int MODE>
__global__ void __launch_bounds__(256, 4) k_raster(RasterArgs A) {
  if (A.ctr->skip_raster) return;
  using SP = Split<MODE>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned* acc32 = reinterpret_cast<unsigned*>(smem_raw);
  long long* acc64 = reinterpret_cast<long long*>(smem_raw);
  float* accf = reinterpret_cast<float*>(smem_raw);
  Staged* stage_all = reinterpret_cast<Staged*>(smem_raw + RasterSmem<MODE>::acc_words * 4);
  uint8_t* owner_all = reinterpret_cast<uint8_t*>(stage_all + 8 * 32);
  int* pref_all = reinterpret_cast<int*>(owner_all + 8 * 1024);
  __shared__ unsigned long long s_unit;
  // F32: the windows below the first that the unit has terms in (bit w); per channel 2^(bits - E), the
  // scale of the first window's split
  __shared__ unsigned s_below;
  __shared__ float s_scale[4];
  if (MODE == RM_F32 && threadIdx.x < 4) s_scale[threadIdx.x] = pow2f(SP::bits - term_exponent(A, threadIdx.x));
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const unsigned acc_addr = (unsigned)__cvta_generic_to_shared(acc32);
  Staged* stage = stage_all + warp * 32;
  uint8_t* owner = owner_all + warp * 1024;
  int* pref = pref_all + warp * 33;
  const BlendDev& B = A.blend;
  uint32_t my_pixels = 0;
  unsigned long long n_units = A.ctr->units;
  if (n_units > A.units_cap) n_units = A.units_cap;
  if (SP::on) {  // the planes start at zero, and every flush leaves them so
    uint4* z = reinterpret_cast<uint4*>(acc32);
    for (int k = threadIdx.x; k < RasterSmem<MODE>::acc_words / 4; k += blockDim.x) z[k] = make_uint4(0, 0, 0, 0);
  }
  for (;;) {
    if (threadIdx.x == 0) {
      s_unit = atomicAdd(&A.ctr->unit_cursor, 1ull);
      if (MODE == RM_F32) s_below = 0u;
    }
    __syncthreads();
    const unsigned long long u = s_unit;
    if (u >= n_units) break;
    const Unit U = A.units[u];
    const CanvasLoc C = canvas_of_bin(A, U.tile);
    const uint32_t lbin = (uint32_t)(U.tile - C.bin_base);
    const uint32_t tile = lbin >> 1;
    const bool xmajor = (lbin & 1u) == 0;
    const uint32_t tx = tile % C.ntx, ty = tile / C.ntx;
    const int tm = xmajor ? (int)tx : (int)ty, tn = xmajor ? (int)ty : (int)tx;
    const int nmin = (int)(xmajor ? C.H : C.W);
    // minor pixels of the tile: floor(v) in [tn TILE, hi) exactly when v is
    const float vlo = (float)(tn * TILE), vhi = (float)min(tn * TILE + TILE, nmin);
    if (MODE == RM_FIXED_MINMAX) {
      for (int k = threadIdx.x; k < 4 * TILE_PX; k += blockDim.x) acc64[k] = ident64(B.op[k / TILE_PX]);
    } else if (!SP::on) {
      for (int k = threadIdx.x; k < 4 * TILE_PX; k += blockDim.x) accf[k] = ident32(B.op[k / TILE_PX]);
    }
    if (!SP::on) __syncthreads();
    // Adds one staged segment's terms to a cell of the tile when on.  Split sums take no branch
    // (eight predicated atomics cost a branch each): a lane that is off adds zeros to the cell
    // of its own bank in row 0.  alpha_c: some alpha term of the batch has a low part (an alpha
    // of 1, the usual one, has none).
    auto deposit = [&](const uint4& q0, const uint4& q1, int cell, bool on, bool alpha_c) {
      const unsigned qs[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
      if (SP::on) {
        const unsigned a = acc_addr + 4u * (unsigned)(on ? cell : (int)lane), m = on ? 0xffffffffu : 0u;
#pragma unroll
        for (int w = 0; w < 8; ++w)
          if (w != 6 || alpha_c) shared_add(a + 4u * PLANE * w, qs[w] & m);
      } else if (on) {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          const int op = B.op[ch];
          if (MODE == RM_FIXED_MINMAX) {
            const long long q = (long long)(((unsigned long long)qs[2 * ch + 1] << 32) | qs[2 * ch]);
            long long* p = acc64 + ch * TILE_PX + cell;
            if (op == LG_BO_MIN) atomicMin(p, q);
            else if (op == LG_BO_MAX) atomicMax(p, q);
            else atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)q);
          } else {
            const float v = __uint_as_float(qs[ch]);
            float* pf = accf + ch * TILE_PX + cell;
            if (op == LG_BO_MIN || op == LG_BO_MAX) f32_minmax(pf, v, op == LG_BO_MIN);
            else atomicAdd(pf, v);
          }
        }
      }
    };
    const uint64_t end = min(U.begin + U.n, A.refs_cap);
    for (int pass = 0;;) {  // F32: the windows of terms; else once
      const float pass_scale = MODE == RM_F32 ? pow2f(F32_WINDOW * pass) : 1.0f;
      const uint32_t counted = MODE == RM_F32 && pass ? 0u : 1u;
      uint32_t next_ref = 0;  // a batch ahead: the segments' addresses do not wait for the list
      if (U.begin + (uint64_t)warp * 32 + lane < end) next_ref = A.refs[U.begin + (uint64_t)warp * 32 + lane];
      for (uint64_t base = U.begin + (uint64_t)warp * 32; base < end; base += (uint64_t)nwarps * 32) {
        // lane-parallel: fetch 32 segments, set them up and clip them to this tile
        const uint64_t r = base + lane;
        const uint32_t si = next_ref;
        if (r + (uint64_t)nwarps * 32 < end) next_ref = A.refs[r + (uint64_t)nwarps * 32];
        Staged st;
        st.mask = 0;
        int c0 = 0, cnt = 0;
        // F32: the pass's window of scaled magnitudes; terms elsewhere; their windows; those for the image
        constexpr float top = (float)(1 << SP::bits), low = top / (1 << F32_WINDOW);
        bool outside = false;
        unsigned below = 0, big = 0;
        float term[4];
        if (r < end) {
          const float4* sp = reinterpret_cast<const float4*>(A.segs + si);
          const float4 g = __ldg(sp), cc = __ldg(sp + 1);
          lg_segment sg;
          sg.x0 = g.x; sg.y0 = g.y; sg.x1 = g.z; sg.y1 = g.w;
          sg.color[0] = cc.x; sg.color[1] = cc.y; sg.color[2] = cc.z; sg.color[3] = cc.w;
          RSetup R;
          if (raster_setup(sg, C.W, C.H, R)) {
            c0 = max(R.lo - tm * TILE, 0);
            cnt = max(min(R.hi - tm * TILE, TILE) - c0, 0);
            st.ua = R.ua; st.va = R.va; st.slope = R.slope;
            if (cnt > 0) st.mask = (cnt >= 32 ? 0xffffffffu : (1u << cnt) - 1u) << c0;
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {
              const float v = contribution(B, ch, sg.color);
              const bool neg = B.op[ch] == LG_BO_REVERSE_SUBTRACT;
              term[ch] = neg ? -v : v;
              if (MODE == RM_F32) {
                const float m = fabsf(v), t = m * (s_scale[ch] * pass_scale);
                const bool in = t >= low && t < top;
                split_bits<MODE>(in ? t : 0.0f, (v < 0.0f) != neg, st.q[2 * ch], st.q[2 * ch + 1]);
                outside |= !in && m != 0.0f;
              } else if (MODE == RM_FIXED_SPLIT) {
                if (!split_fixed(v, neg, st.q[2 * ch], st.q[2 * ch + 1])) big = 15u;
              } else if (MODE == RM_FIXED_MINMAX) {
                long long q = to_fixed(v);
                if (neg) q = -q;
                st.q[2 * ch] = (unsigned)(q & 0xffffffffll);
                st.q[2 * ch + 1] = (unsigned)(q >> 32);
              } else {
                st.q[ch] = __float_as_uint(term[ch]);
              }
            }
            if (MODE == RM_F32 && pass == 0 && outside) {
              static_assert(F32_PASSES == 3, "two windows below the first");
#pragma unroll
              for (int ch = 0; ch < 4; ++ch) {
                const float m = fabsf(term[ch]), t = m * s_scale[ch];
                if (m == 0.0f || (t >= low && t < top)) continue;
                if (!(t < top) || t < low / ((float)(1 << F32_WINDOW) * (1 << F32_WINDOW))) big |= 1u << ch;
                else below |= t < low / (1 << F32_WINDOW) ? 4u : 2u;
              }
            }
          }
        }
        if (MODE == RM_F32) {
          if (pass == 0) {
            const unsigned all = __reduce_or_sync(0xffffffffu, cnt > 0 ? below : 0u);
            if (all && lane == 0) atomicOr(&s_below, all);
          } else if ((st.q[0] | st.q[1] | st.q[2] | st.q[3] | st.q[4] | st.q[5] | st.q[6] | st.q[7]) == 0u) {
            cnt = 0;
          }
        }
        if (SP::on) {  // rare: terms outside the splits' range go straight into the image
          unsigned bigs = __ballot_sync(0xffffffffu, big && cnt > 0);
          if (MODE == RM_FIXED_SPLIT && big) cnt = 0;
          while (bigs) {
            const int k = __ffs(bigs) - 1;
            bigs &= bigs - 1;
            const float bua = __shfl_sync(0xffffffffu, st.ua, k), bva = __shfl_sync(0xffffffffu, st.va, k);
            const float bsl = __shfl_sync(0xffffffffu, st.slope, k);
            const unsigned bm = __shfl_sync(0xffffffffu, st.mask, k), bch = __shfl_sync(0xffffffffu, big, k);
            const int i = tm * TILE + (int)lane;
            const float v = __fmaf_rn(__fsub_rn(__fadd_rn((float)i, 0.5f), bua), bsl, bva);
            const bool on = ((bm >> lane) & 1u) && v >= vlo && v < vhi;
            const int j = on ? (int)v : 0;
            const uint32_t x = xmajor ? (uint32_t)i : (uint32_t)j, y = xmajor ? (uint32_t)j : (uint32_t)i;
            const uint64_t px = (C.px_base + (uint64_t)y * C.W + x) * 4;
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {
              const float tv = __shfl_sync(0xffffffffu, term[ch], k);
              if (!on || !((bch >> ch) & 1u)) continue;
              if (MODE == RM_F32) {
                image_add(A, px + ch, (double)tv);
              } else {
                const long long q = to_fixed(tv);
                if (q) atomicAdd(reinterpret_cast<unsigned long long*>(A.accum) + px + ch, (unsigned long long)q);
              }
            }
            if (MODE == RM_FIXED_SPLIT) my_pixels += on ? 1u : 0u;
          }
        }
        // the batch's segments with columns here, side by side in the warp's stage
        const unsigned drawn = __ballot_sync(0xffffffffu, cnt > 0);
        const int n_drawn = __popc(drawn), pos = __popc(drawn & lanemask_lt());
        const int total = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
        const bool alpha_c = SP::on && __any_sync(0xffffffffu, cnt > 0 && st.q[6] != 0u);
        bool by_lane = total >= LG_RASTER_LANE_MIN * n_drawn;
        // The usual batch: colour terms in [0, 1), whose split parts are the bits of one word each, and
        // one alpha term for all without a low part (an alpha of 1).  Its staged rows take two
        // 16-byte reads instead of three, and reads are a third of the shared-memory traffic.
        if (MODE == RM_FIXED_SPLIT && by_lane && drawn) {
          const unsigned alpha = __shfl_sync(0xffffffffu, st.q[7], __ffs(drawn) - 1);
          const bool wide = cnt > 0 && (st.q[6] != 0u || st.q[7] != alpha || (st.q[1] | st.q[3] | st.q[5]) >> (32 - SP::bits) != 0u ||
                                        (st.q[0] | st.q[2] | st.q[4]) >> SP::bits != 0u);
          if (!__any_sync(0xffffffffu, wide)) {
            uint4* rows = reinterpret_cast<uint4*>(stage);
            if (cnt > 0) {
              rows[2 * pos] = make_uint4(__float_as_uint(st.ua), __float_as_uint(st.va), __float_as_uint(st.slope), st.mask);
              rows[2 * pos + 1] = make_uint4(st.q[0] | st.q[1] << SP::bits, st.q[2] | st.q[3] << SP::bits,
                                             st.q[4] | st.q[5] << SP::bits, 0u);
            }
            __syncwarp();
            const float fi = __fadd_rn((float)(tm * TILE + (int)lane), 0.5f);
            const int cell0 = (int)lane - tn * TILE_PX;
            const unsigned bit = 1u << lane, low = (1u << SP::bits) - 1u;
#pragma unroll 2
            for (int k = 0; k < n_drawn; ++k) {
              const uint4 h = rows[2 * k], q = rows[2 * k + 1];
              const float v = __fmaf_rn(__fsub_rn(fi, __uint_as_float(h.x)), __uint_as_float(h.z), __uint_as_float(h.y));
              const bool on = (h.w & bit) && v >= vlo && v < vhi;
              const unsigned a = acc_addr + 4u * (unsigned)(on ? (int)v * TILE + cell0 : (int)lane), m = on ? 0xffffffffu : 0u;
              const unsigned qr = q.x & m, qg = q.y & m, qb = q.z & m;
              shared_add(a, qr & low);
              shared_add(a + 4u * PLANE, qr >> SP::bits);
              shared_add(a + 8u * PLANE, qg & low);
              shared_add(a + 12u * PLANE, qg >> SP::bits);
              shared_add(a + 16u * PLANE, qb & low);
              shared_add(a + 20u * PLANE, qb >> SP::bits);
              shared_add(a + 28u * PLANE, alpha & m);
              my_pixels += on ? 1u : 0u;
            }
            __syncwarp();
            continue;
          }
        }
        if (cnt > 0) stage[pos] = st;
        if (by_lane) {
          __syncwarp();
          const float fi = __fadd_rn((float)(tm * TILE + (int)lane), 0.5f);
          const int cell0 = (int)lane - tn * TILE_PX;
          const unsigned bit = 1u << lane;
          auto draw = [&](auto low_alpha) {
#pragma unroll 2
            for (int k = 0; k < n_drawn; ++k) {
              const Staged& sk = stage[k];
              const float4 h = *reinterpret_cast<const float4*>(&sk);
              const uint4 q0 = *reinterpret_cast<const uint4*>(&sk.q[0]);
              const uint4 q1 = *reinterpret_cast<const uint4*>(&sk.q[4]);
              const float v = __fmaf_rn(__fsub_rn(fi, h.x), h.z, h.y);
              const bool on = (__float_as_uint(h.w) & bit) && v >= vlo && v < vhi;
              deposit(q0, q1, (int)v * TILE + cell0, on, decltype(low_alpha)::value);
              my_pixels += on ? counted : 0u;
            }
          };
          if (alpha_c) draw(std::true_type{}); else draw(std::false_type{});
        } else {
          // every (segment, pixel column) pair of the batch densely over the lanes
          int incl = cnt;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += y;
          }
          if (cnt > 0) pref[pos] = incl - cnt - c0;  // pair number less the column
          for (int k = 0; k < cnt; ++k) owner[incl - cnt + k] = (uint8_t)pos;
          __syncwarp();
          for (int pi = (int)lane; pi < total; pi += 32) {
            const int k = owner[pi];
            const Staged& sk = stage[k];
            const int col = pi - pref[k];
            const float fi = __fadd_rn((float)(tm * TILE + col), 0.5f);
            const float v = __fmaf_rn(__fsub_rn(fi, sk.ua), sk.slope, sk.va);
            if (!(v >= vlo && v < vhi)) continue;
            deposit(*reinterpret_cast<const uint4*>(&sk.q[0]), *reinterpret_cast<const uint4*>(&sk.q[4]),
                    ((int)v - tn * TILE) * TILE + col, true, alpha_c);
            my_pixels += counted;
          }
        }
        __syncwarp();
      }
      __syncthreads();
      const unsigned rest = MODE == RM_F32 ? s_below >> (pass + 1) : 0u;
      if (SP::on) {
        // flush: four lanes per pixel, one channel each, so that a warp's atomics cover whole
        // 32 B sectors of the image
        // 2^-bits over the scale, by the exponents
        const int scale_exp = MODE == RM_F32 ? (__float_as_int(s_scale[threadIdx.x & 3] * pass_scale) >> 23) - 127 : 0;
        const double unit = __hiloint2double((1023 - scale_exp - SP::bits) << 20, 0);
        for (int k = threadIdx.x; k < 4 * TILE_PX; k += blockDim.x) {
          const int ch = k & 3, cell = k >> 2;
          const int major = cell % TILE, minor = cell / TILE;
          const uint32_t x = tx * TILE + (xmajor ? major : minor), y = ty * TILE + (xmajor ? minor : major);
          unsigned* plane = acc32 + 2 * ch * PLANE + cell;
          const unsigned lo = plane[0], hi = plane[PLANE];
          if ((lo | hi) == 0u) continue;
          plane[0] = 0u;
          plane[PLANE] = 0u;
          const long long q = (long long)(int)hi * (1ll << SP::bits) + (long long)(int)lo;
          if (q == 0 || x >= C.W || y >= C.H) continue;
          const uint64_t px = (C.px_base + (uint64_t)y * C.W + x) * 4;
          if (MODE == RM_F32)
            image_add(A, px + ch, __dmul_rn(__ll2double_rn(q), unit));  // both steps exact
          else
            atomicAdd(reinterpret_cast<unsigned long long*>(A.accum) + px + ch, (unsigned long long)q);
        }
      } else {
        // flush: one global atomic per touched pixel channel
        for (int k = threadIdx.x; k < TILE_PX; k += blockDim.x) {
          const int row = k / TILE, col = k % TILE;
          const uint32_t x = tx * TILE + col, y = ty * TILE + row;
          if (x >= C.W || y >= C.H) continue;
          const uint64_t px = (C.px_base + (uint64_t)y * C.W + x) * 4;
          const int cell = xmajor ? row * TILE + col : col * TILE + row;
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            const int op = B.op[ch];
            if (MODE == RM_FIXED_MINMAX) {
              const long long v = acc64[ch * TILE_PX + cell];
              if (v == ident64(op)) continue;
              long long* g = reinterpret_cast<long long*>(A.accum) + px + ch;
              if (op == LG_BO_MIN) atomicMin(g, v);
              else if (op == LG_BO_MAX) atomicMax(g, v);
              else atomicAdd(reinterpret_cast<unsigned long long*>(g), (unsigned long long)v);
            } else {
              const float v = accf[ch * TILE_PX + cell];
              if (v == ident32(op)) continue;
              float* g = reinterpret_cast<float*>(A.accum) + px + ch;
              if (op == LG_BO_MIN || op == LG_BO_MAX) f32_minmax(g, v, op == LG_BO_MIN);
              else atomicAdd(g, v);
            }
          }
        }
      }
      __syncthreads();
      if (rest == 0u) break;
      pass += __ffs(rest);
    }
  }
  add_block_counts<1>({my_pixels}, {&A.ctr->pixels});
}

// ------------------------------------------------------------------ string-mod lines
// A few thousand lines per frame: one warp per line, one lane per major-axis pixel, and
// each pixel's terms go straight into the image with global atomics (int64 sums and
// min / max are order-independent, so the image stays bit-reproducible in fixed point).
template <bool FIXED>
__global__ void __launch_bounds__(256) k_raster_chords(RasterArgs A, const lg_chord* chords, uint64_t n) {
  const unsigned lane = lane_id();
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const BlendDev& B = A.blend;
  const float sc = (float)A.H * 0.5f, cx = (float)A.W * 0.5f;
  uint32_t my_pixels = 0;
  for (uint64_t k = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; k < n; k += nw) {
    const lg_chord c = chords[k];
    lg_segment sg;
    sg.x0 = c.x0; sg.y0 = c.y0; sg.x1 = c.x1; sg.y1 = c.y1;
    RSetup R;
    if (!raster_setup(sg, A.W, A.H, R)) continue;
    // the vertices' major coordinates before raster_setup orders them
    const float U0 = R.xmajor ? __fmaf_rn(c.x0, sc, cx) : __fmaf_rn(-c.y0, sc, sc);
    const float dU = __fsub_rn(R.xmajor ? __fmaf_rn(c.x1, sc, cx) : __fmaf_rn(-c.y1, sc, sc), U0);
    float dc[4];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) dc[ch] = __fsub_rn(c.color1[ch], c.color0[ch]);
    const int nmin = (int)(R.xmajor ? A.H : A.W);
    for (int i = R.lo + (int)lane; i < R.hi; i += 32) {
      const int j = raster_minor(R, i);
      if (j < 0 || j >= nmin) continue;
      float f = __fdiv_rn(__fsub_rn(__fadd_rn((float)i, 0.5f), U0), dU);
      f = fminf(fmaxf(f, 0.0f), 1.0f);
      float src[4];
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) src[ch] = __fmaf_rn(f, dc[ch], c.color0[ch]);
      const uint32_t x = R.xmajor ? (uint32_t)i : (uint32_t)j, y = R.xmajor ? (uint32_t)j : (uint32_t)i;
      const uint64_t px = ((uint64_t)y * A.W + x) * 4;
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) {
        const int op = B.op[ch];
        const float v = contribution(B, ch, src);
        if (FIXED) {
          long long q = to_fixed(v);
          long long* g = reinterpret_cast<long long*>(A.accum) + px + ch;
          if (op == LG_BO_MIN) atomicMin(g, q);
          else if (op == LG_BO_MAX) atomicMax(g, q);
          else {
            if (op == LG_BO_REVERSE_SUBTRACT) q = -q;
            if (q) atomicAdd(reinterpret_cast<unsigned long long*>(g), (unsigned long long)q);
          }
        } else {
          float* g = reinterpret_cast<float*>(A.accum) + px + ch;
          if (op == LG_BO_MIN || op == LG_BO_MAX) {
            float o = *g;
            while (op == LG_BO_MIN ? v < o : v > o) {
              const float w = __int_as_float(atomicCAS(reinterpret_cast<int*>(g), __float_as_int(o), __float_as_int(v)));
              if (w == o) break;
              o = w;
            }
          } else {
            image_add(A, px + ch, op == LG_BO_REVERSE_SUBTRACT ? -v : v);
          }
        }
      }
      ++my_pixels;
    }
  }
  add_block_counts<1>({my_pixels}, {&A.ctr->pixels});
}

template __global__ void k_raster_chords<true>(RasterArgs A, const lg_chord* chords, uint64_t n);
template __global__ void k_raster_chords<false>(RasterArgs A, const lg_chord* chords, uint64_t n);

static void (*raster_kernel(int mode))(RasterArgs) {
  switch (mode) {
    case RM_FIXED_SPLIT_: return k_raster<RM_FIXED_SPLIT>;
    case RM_FIXED_MINMAX_: return k_raster<RM_FIXED_MINMAX>;
    case RM_F32_: return k_raster<RM_F32>;
    default: return k_raster<RM_F32_MINMAX>;
  }
}
static int raster_smem_bytes(int mode) {
  switch (mode) {
    case RM_FIXED_SPLIT_: return RasterSmem<RM_FIXED_SPLIT>::bytes;
    case RM_FIXED_MINMAX_: return RasterSmem<RM_FIXED_MINMAX>::bytes;
    case RM_F32_: return RasterSmem<RM_F32>::bytes;
    default: return RasterSmem<RM_F32_MINMAX>::bytes;
  }
}

cudaError_t raster_occupancy(int mode, int* occ) {
  cudaError_t e = cudaFuncSetAttribute(raster_kernel(mode), cudaFuncAttributeMaxDynamicSharedMemorySize, raster_smem_bytes(mode));
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, raster_kernel(mode), 256, (size_t)raster_smem_bytes(mode));
  return e;
}

void launch_raster(int mode, int grid, cudaStream_t stream, const RasterArgs& A) {
  raster_kernel(mode)<<<grid, 256, (size_t)raster_smem_bytes(mode), stream>>>(A);
}

uint32_t raster_unit_refs(int mode) { return mode == RM_F32_ ? F32_UNIT_REFS : SPLIT_UNIT_REFS; }

// ------------------------------------------------------------------ resolve
__device__ __forceinline__ float4 load_px(const void* acc, int kind, uint64_t i) {
  if (kind == ACC_F64) {
    const double4_32a v = reinterpret_cast<const double4_32a*>(acc)[i];
    return make_float4(__double2float_rn(v.x), __double2float_rn(v.y), __double2float_rn(v.z), __double2float_rn(v.w));
  }
  if (kind == ACC_I64) {
    const longlong4_32a v = reinterpret_cast<const longlong4_32a*>(acc)[i];
    const float s = 2.3283064365386963e-10f;  // 2^-32
    return make_float4(__fmul_rn(__ll2float_rn(v.x), s), __fmul_rn(__ll2float_rn(v.y), s),
                       __fmul_rn(__ll2float_rn(v.z), s), __fmul_rn(__ll2float_rn(v.w), s));
  }
  return reinterpret_cast<const float4*>(acc)[i];
}

__global__ void k_resolve_f16(const void* acc, int kind, uint32_t W, uint32_t H, uint16_t* dst, size_t pitch) {
  const uint64_t n = (uint64_t)W * H;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const float4 f = load_px(acc, kind, i);
    const uint32_t y = (uint32_t)(i / W), x = (uint32_t)(i % W);
    ushort4 h;
    h.x = __half_as_ushort(__float2half_rn(f.x));
    h.y = __half_as_ushort(__float2half_rn(f.y));
    h.z = __half_as_ushort(__float2half_rn(f.z));
    h.w = __half_as_ushort(__float2half_rn(f.w));
    *reinterpret_cast<ushort4*>(reinterpret_cast<char*>(dst) + y * pitch + (uint64_t)x * 8) = h;
  }
}

// renderer.rs:313-328: u8 = (f16 value ^ (1 / 2.2) * 255) as u8 (saturating, truncating)
__global__ void k_resolve_rgba8(const void* acc, int kind, uint32_t W, uint32_t H, uint8_t* dst, size_t pitch) {
  const uint64_t n = (uint64_t)W * H;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const float4 f = load_px(acc, kind, i);
    const uint32_t y = (uint32_t)(i / W), x = (uint32_t)(i % W);
    const float c[4] = {f.x, f.y, f.z, f.w};
    uchar4 o;
    unsigned char* po = &o.x;
    for (int k = 0; k < 4; ++k) {
      const float h = __half2float(__float2half_rn(c[k]));
      const float g = __fmul_rn(powf(h, __fdiv_rn(1.0f, 2.2f)), 255.0f);
      po[k] = (g != g || g <= 0.0f) ? 0 : (g >= 255.0f ? 255 : (unsigned char)g);
    }
    *reinterpret_cast<uchar4*>(dst + y * pitch + (uint64_t)x * 4) = o;
  }
}

}  // namespace lgd
