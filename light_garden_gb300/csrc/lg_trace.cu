// lg_trace.cu — ray generation and the per-generation trace kernels (sm_103a).
//
// Tracer::trace (src/light_garden/tracer.rs:360-493) walks a breadth-first ray tree per
// primary ray.  Here each generation of all trees of all lights is one device queue (a
// wavefront), processed by a short chain of kernels so that warps stay full no matter how
// the trees branch:
//   gen 0 reads a virtual queue (light, ray index) and generates the primary ray
//   (light.rs:103-115, 163-174, 225-249); gen g > 0 reads the queue written by gen g-1.
//   For each ray: cutoff (tracer.rs:378-384), nearest hit (412-424), medium (428-442),
//   refract / reflect with colour split (444-481) or canvas exit (482-488).
//   Segments are appended to the segment ring and children to the next queue with one
//   atomic per warp (ballot + popc compaction).
// The chain per generation (k_scan, k_refine over 4 leaf-kind lists, k_full, k_bounce) is
// described above k_scan below.
#include "lg_kernels.cuh"
#include "lg_trace_common.cuh"

namespace lgd {

// ------------------------------------------------------------------- primary rays
// native FP64 (only here): the reference's f64 sin_cos / atan per primary ray
__device__ inline void primary_ray(const LightDev& L, uint64_t i, double& ox, double& oy, double& dx, double& dy) {
  const double n = (double)L.num_rays;
  if (L.kind == LG_LIGHT_POINT) {  // light.rs:168-172
    const double f = (double)i * 3.141592653589793 * 2.0 / n;
    double s, c;
    sincos(f, &s, &c);
    ox = L.ox; oy = L.oy; dx = c; dy = s;
  } else if (L.kind == LG_LIGHT_SPOT) {  // light.rs:230-247
    const double sx = L.vx, sy = L.vy;
    const double dir_angle =
        fabs(sx) < SPOT_EPSILON ? (sy >= 0.0 ? 3.141592653589793 * 0.5 : -3.141592653589793 * 0.5) : atan(sy / sx);
    const double min_angle = dir_angle - 0.5 * L.spot_angle;
    const double ang = min_angle + ((double)(i + 1) / n) * L.spot_angle;
    double s, c;
    sincos(ang, &s, &c);
    const double sign = signbit(sx) ? -1.0 : 1.0;
    ox = L.ox; oy = L.oy; dx = sign * c; dy = sign * s;
  } else {  // directional: origins along a -> b, unit left normal
    const double ex = L.vx - L.ox, ey = L.vy - L.oy;
    const double r = (double)i / n;
    ox = L.ox + ex * r;
    oy = L.oy + ey * r;
    const double l = sqrt(ey * ey + ex * ex);
    dx = l > 0.0 ? -ey / l : -ey;
    dy = l > 0.0 ? ex / l : ex;
  }
}

// Start media (tracer.rs:280-287: the last object that contains the light wins), a warp per
// light: see k_light_setup_x.
template <bool MULTI>
__global__ void k_light_setup(SceneDev S) {
  const uint32_t l0 = S.serve ? S.light_lo : 0u, l1 = S.serve ? S.light_hi : S.n_lights;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t l = l0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); l < l1; l += warps) {
    LightDev& L = S.lights[l];
    const SceneLoc sl = scene_of<MULTI>(S, L.scene);
    const df px = df_from_double(L.ox), py = df_from_double(L.oy);
    const uint32_t k = last_object_of_warp(sl.base, sl.n, [&](uint32_t j) {
      bool near = false;
      return (S.info[j].flags & INFO_MATERIAL) && obj_contains64(S, j, px, py, near, 0.0f);
    });
    if (lane_id() == 0) L.n0 = k == 0xffffffffu ? DF_ONE : S.info[k].n;
  }
}
template __global__ void k_light_setup<false>(SceneDev);
template __global__ void k_light_setup<true>(SceneDev);

// ------------------------------------------------------------------- one generation
// Each generation runs as four kernels over the generation's queue (a wavefront), so that
// every kernel executes one compact code path on coherent work:
//   k_scan     FP32: nearest-hit search bound and candidate list per ray; sorts the rays
//              into work lists (refine circle / rect / segment, full solve)
//   k_refine   double-float refinement of a winner the FP32 scan proved (the leaf-kind
//              lists one after the other)
//   k_full     double-float solve of every candidate (near ties, uncertain roots, cubic
//              and deep CSG objects), grouped by solve class
//   k_bounce   medium (tracer.rs:428-442), refract / reflect with colour split
//              (444-481) or canvas exit (482-488); appends segments and children
__device__ __forceinline__ int leaf_kind_of(uint32_t info, int leaf) {
  return (int)(leaf == 0 ? info_leaf_a(info) : info_leaf_b(info));
}

// appends idx to work list `list` (-1: none) with one atomic per (warp, list)
__device__ __forceinline__ void list_append(const TraceBufs& B, uint32_t gen, int list, uint32_t idx) {
  const unsigned act = __activemask();
  const unsigned grp = __match_any_sync(act, list);
  if (list < 0) return;
  const int leader = __ffs(grp) - 1;
  unsigned long long base = 0;
  if ((int)lane_id() == leader) base = atomicAdd(&B.ctr->list_count[gen][list], (unsigned long long)__popc(grp));
  base = __shfl_sync(grp, base, leader);
  const unsigned long long slot = base + __popc(grp & lanemask_lt());
  if (slot < B.queue_cap) B.list[list][slot] = idx;
}

// Canvas exit of a ray that hits no object, when its origin is clearly inside the canvas
// and the exit is clearly not at a corner: the exit face is found in FP32, the exit point
// computed in double-float.  Anything else takes the precise path in k_bounce.
__device__ __forceinline__ bool fast_canvas_exit(const df aspect, const RayRec& r, float& x1, float& y1, float& L) {
  const float ax = aspect.hi, ox = r.ox.hi, oy = r.oy.hi, dx = r.dx.hi, dy = r.dy.hi;
  if (!(fabsf(ox) < ax - 1e-4f && fabsf(oy) < 1.0f - 1e-4f)) return false;
  const float tx = dx > 0.0f ? (ax - ox) / dx : dx < 0.0f ? (-ax - ox) / dx : INFINITY;
  const float ty = dy > 0.0f ? (1.0f - oy) / dy : dy < 0.0f ? (-1.0f - oy) / dy : INFINITY;
  if (!(fabsf(tx - ty) > 1e-4f * (fminf(tx, ty) + 1.0f))) return false;
  df t;
  if (tx < ty) {
    const df bound = dx > 0.0f ? aspect : -aspect;
    t = (bound - r.ox) / r.dx;
  } else {
    const df bound = dy > 0.0f ? DF_ONE : -DF_ONE;
    t = (bound - r.oy) / r.dy;
  }
  x1 = (r.ox + r.dx * t).hi;
  y1 = (r.oy + r.dy * t).hi;
  L = r.ex + t.hi * r.ea;
  return true;
}

// the segment of an emitting lane at its place in the ring
__device__ __forceinline__ void store_segment(const SceneDev& S, const TraceBufs& B, const RayRec& r, float x1, float y1,
                                              uint8_t flags, int hit, unsigned long long slot, uint32_t& my_near,
                                              uint32_t& my_ill) {
  if (flags & LG_PATH_NEAR_DEGENERATE) ++my_near;
  if (flags & LG_PATH_ILL_CONDITIONED) ++my_ill;
  if (slot >= B.seg_cap) return;
  float4* dst = reinterpret_cast<float4*>(B.segs + slot);
  dst[0] = make_float4(r.ox.hi, r.oy.hi, x1, y1);
  dst[1] = make_float4(r.c[0], r.c[1], r.c[2], r.c[3]);
  if (B.seg_scene) B.seg_scene[slot] = r.scene;
  if (S.record_paths) {
    lg_path_record pr;
    pr.path = r.path; pr.primary = r.prim; pr.light = r.light; pr.gen = r.gen;
    pr.flags = flags; pr.hit = hit; pr.source = LG_SRC_TRACE;
    B.paths[slot] = pr;
  }
}

// appends one segment per emitting lane with one atomic per warp (all lanes call)
__device__ __forceinline__ void emit_segments(const SceneDev& S, const TraceBufs& B, bool emit, const RayRec& r,
                                              float x1, float y1, uint8_t flags, int hit,
                                              uint32_t& my_near, uint32_t& my_ill) {
  const unsigned emask = __ballot_sync(0xffffffffu, emit);
  if (!emask) return;
  unsigned long long sbase = 0;
  const int leader = __ffs(emask) - 1;
  if ((int)lane_id() == leader) sbase = atomicAdd(&B.ctr->seg_count, (unsigned long long)__popc(emask));
  sbase = __shfl_sync(0xffffffffu, sbase, leader);
  if (emit) store_segment(S, B, r, x1, y1, flags, hit, sbase + __popc(emask & lanemask_lt()), my_near, my_ill);
}

// Warp-cooperative FP32 scan.  Every lane bounding-tests its own ray against a run of
// objects (pruned by its running bound thr) and writes the passing (ray, object) pairs to
// the warp's shared buffer; then all 32 lanes classify the warp's pairs side by side, so
// the exact FP32 tests run at full SIMD width instead of only in the lanes whose ray
// happens to cross a given object.  Each lane then folds its own results: thr shrinks
// with every certain hit and the candidates (key <= thr) go to the precise solve, which
// applies the first-in-object-order tie rule of tracer.rs:404,417 itself.  The runs are
// either the object table in chunks of SCAN_CHUNK, or (culling grid) the objects listed
// in the grid cells the lane's ray crosses, nearest cell first.
// Launch shape.  The pair slots per lane between classifications (CHUNK, 8 or 16) are a
// template parameter (scan_pairs_of says when which).  CTAs per SM of the culled scan
// and its cell steps between classifications are build-time (-DLG_SCAN_CULL_BLOCKS=...,
// -DLG_SCAN_WALK_CELLS=..., for sweeps).
#ifndef LG_SCAN_CULL_BLOCKS
#define LG_SCAN_CULL_BLOCKS 4
#endif
#ifndef LG_SCAN_WALK_CELLS
#define LG_SCAN_WALK_CELLS 8
#endif
constexpr int SCAN_WARPS = 4;
constexpr int WALK_CELLS = LG_SCAN_WALK_CELLS;  // culled scan: cell steps between classifications (2 to 16: within 2 %)
constexpr int SCAN_CULL_BLOCKS = LG_SCAN_CULL_BLOCKS;  // culled scan: CTAs per SM the registers are sized for

struct __align__(16) PairSlot {
  float key, ub, s;
  uint32_t m;  // object | (leaf + 1) << 16 | (face + 1) << 24; before classification key holds lb
};

template <int CHUNK>
struct ScanSmemT {  // [slot][lane]: a warp's 32 lanes touch 32 consecutive slots
  PairSlot pairs[SCAN_WARPS][CHUNK][32];
  PairSlot cand[SCAN_WARPS][CAND][32];
  float4 ray[SCAN_WARPS][32];
  uint32_t src[SCAN_WARPS][32];
  uint32_t base[SCAN_WARPS][32];
  union {
    uint16_t pair[CHUNK <= 8 ? CHUNK * 32 : 1];  // slot order: the lane and slot of every pair
    int off[32];                                 // lane order: where a lane's pairs start
  } map[SCAN_WARPS];
};

int scan_smem_bytes(int pairs) { return pairs <= 8 ? (int)sizeof(ScanSmemT<8>) : (int)sizeof(ScanSmemT<16>); }

template <bool MULTI, bool CULL, bool EXACT, int CHUNK>
__global__ void __launch_bounds__(SCAN_WARPS * 32, CULL ? SCAN_CULL_BLOCKS : 4)
    k_scan(SceneDev S, TraceBufs B, uint32_t gen, int smem_fits) {
  constexpr int SCAN_CHUNK = CHUNK;
  using ScanSmem = ScanSmemT<SCAN_CHUNK>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  ScanSmem& W = *reinterpret_cast<ScanSmem*>(smem_raw);
  ObjScan* sobj = reinterpret_cast<ObjScan*>(smem_raw + sizeof(ScanSmem));
  stamp_start(B.ctr, gen, 0);
  const uint64_t n_real = n_real_of(S, B, gen);
  const uint64_t n_in = n_in_of(S, B, gen);
  if ((uint64_t)blockIdx.x * blockDim.x >= n_in) return;  // no ray for this CTA
  __shared__ uint32_t cls_count[SCAN_WARPS];  // classifications, one count per warp
  if (lane_id() == 0) cls_count[threadIdx.x >> 5] = 0;
  __syncwarp();
  uint32_t my_visits = 0, my_near = 0, my_ill = 0;
  uint32_t my_tests = 0;
  bool failed;
  const ObjScan* objs = stage_objects(S, sobj, &bar, !MULTI && smem_fits != 0, B.ctr, failed);
  if (failed) return;
  RayRec* q = B.queue[gen & 1];
  const unsigned lane = lane_id(), w = threadIdx.x >> 5;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  const bool ordered = MULTI || (B.order && sorts<MULTI>(n_real));
  for (uint64_t base = warp * 32; base < n_in; base += nwarps * 32) {
    // queued rays in visiting order (scene, place, direction), so that a warp's rays (and a
    // CTA's warps) share one scene; new primaries follow, ordered by light
    uint64_t idx = base + lane;
    bool valid = idx < n_in;
    if (ordered && valid && idx < n_real) {
      idx = B.order[idx];
      valid = idx < n_real;
    }
    bool live = valid;
    RayRec r;
    if (live) {
      if (idx >= n_real) {
        const uint64_t v = idx - n_real;  // primary number among this launch's new lights
        uint32_t l = S.serve ? S.light_lo : 0u, lhi = S.serve ? S.light_hi : S.n_lights;
        while (lhi - l > 1) {  // the last light whose first primary is <= v
          const uint32_t mid = (l + lhi) >> 1;
          if (S.lights[mid].first <= v) l = mid; else lhi = mid;
        }
        const LightDev& L = S.lights[l];
        const uint64_t i = S.ray_offset + (uint64_t)S.ray_stride * (v - L.first);
        double pox, poy, pdx, pdy;
        if (EXACT) {  // exact mode: the FP64 coordinates themselves, in the df slots
          lgx::primary_ray_x(L.kind, L.ox, L.oy, L.vx, L.vy, L.spot_angle, L.dir_angle, (double)L.num_rays, i, pox,
                             poy, pdx, pdy);
          r.ox = xdf(pox); r.oy = xdf(poy); r.dx = xdf(pdx); r.dy = xdf(pdy);
        } else {
          primary_ray(L, i, pox, poy, pdx, pdy);
          r.ox = df_from_double(pox); r.oy = df_from_double(poy);
          r.dx = df_from_double(pdx); r.dy = df_from_double(pdy);
        }
        r.medium = MEDIUM_LIGHT;
        r.src_obj = SRC_NONE;
        r.src_leaf = 0;
        r.c[0] = L.color[0]; r.c[1] = L.color[1]; r.c[2] = L.color[2]; r.c[3] = L.color[3];
        r.path = 0;
        r.prim = (uint32_t)i;
        r.light = (uint16_t)(MULTI ? l - S.scenes[L.scene].light_base : l);
        r.gen = 0;
        r.flags = 0;
        r._pad = 0;
        r.scene = MULTI ? (uint16_t)L.scene : (uint16_t)0;
        // rounding of the light's ray generator (sin/cos/atan) and the double-float split
        r.ex = EXACT ? 0.0f : DF_ROUND * (1.0f + fabsf(r.ox.hi) + fabsf(r.oy.hi));
        r.ea = EXACT ? 0.0f : DF_ROUND;
        if (idx < B.queue_cap) q[idx] = r;
      } else {
        r = q[idx];
      }
    }
    const SceneLoc sl = scene_of<MULTI>(S, live ? r.scene : 0u);
    const bool dead = live && below_cutoff(r.c, sl.cutoff);
    live = live && !dead;
    const float ox = EXACT ? (float)xd(r.ox) : r.ox.hi, oy = EXACT ? (float)xd(r.oy) : r.oy.hi;
    const float dx = EXACT ? (float)xd(r.dx) : r.dx.hi, dy = EXACT ? (float)xd(r.dy) : r.dy.hi;
    W.ray[w][lane] = make_float4(ox, oy, dx, dy);
    W.src[w][lane] = live ? ((uint32_t)r.src_obj << 8 | r.src_leaf) : 0xffffffffu;
    W.base[w][lane] = sl.base;
    float thr = 3e38f;  // finite: a certain miss (key INFINITY) is never a candidate
    int nc = 0;
    bool overflow = false;
    // The warp scans one scene at a time: a multi-scene warp (rays of several scenes, at
    // the seams of the queue) runs one pass per distinct scene with that scene's lanes;
    // a single-scene warp runs exactly one pass.
    const unsigned live_mask = __ballot_sync(0xffffffffu, live);
    const uint32_t my_scene = live ? (uint32_t)r.scene : 0xffffffffu;
    unsigned pending = MULTI ? live_mask : (live_mask ? 1u : 0u);
    while (pending) {
      bool mine;
      uint32_t g_lo, g_hi, pass_scene = 0;
      if (MULTI) {
        const int leader = __ffs(pending) - 1;
        pass_scene = __shfl_sync(0xffffffffu, my_scene, leader);
        const unsigned grp = __ballot_sync(0xffffffffu, my_scene == pass_scene);
        pending &= ~grp;
        mine = (grp >> lane) & 1u;
        g_lo = __shfl_sync(0xffffffffu, sl.base, leader);
        g_hi = g_lo + __shfl_sync(0xffffffffu, sl.n, leader);
      } else {
        pending = 0;
        mine = live;
        g_lo = 0;
        g_hi = S.n_obj;
      }
      // Classifies the warp's cnt-per-lane pairs side by side, then folds each lane's own
      // results: thr shrinks with every certain hit, candidates (key <= thr) are kept.
      auto classify_fold = [&](int cnt) {
        constexpr bool SLOT_ORDER = SCAN_CHUNK <= 8;
        int total = 0;
        if constexpr (SLOT_ORDER) {
          // The warp's pairs in slot order, the lanes' first pairs before their second ones: rays
          // of a warp meet the same objects in the same order, so that a pass of 32 pairs has few
          // objects and leaf kinds (CSG frame, 786,432 primaries: scan 90.8 -> 78.3 ms against
          // lane order; each lane its own pairs, uncompacted, 90.2).
          for (int k = 0; k < SCAN_CHUNK; ++k) {
            const unsigned has = __ballot_sync(0xffffffffu, cnt > k);
            if (!has) break;
            if (cnt > k) W.map[w].pair[total + __popc(has & lanemask_lt())] = (uint16_t)(lane | (unsigned)k << 5);
            total += __popc(has);
          }
        } else {
          // lane after lane: the map of 16 slots would cost the fourth CTA of an SM its shared
          // memory (30 CSG objects, 65,536 primaries: 4 % slower)
          int incl = cnt;
  #pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if ((int)lane >= o) incl += y;
          }
          W.map[w].off[lane] = incl - cnt;
          total = __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) cls_count[w] += (uint32_t)total;
        __syncwarp();
        for (int p = (int)lane; p < total; p += 32) {
          int lo, k;
          if constexpr (SLOT_ORDER) {
            const int at = W.map[w].pair[p];
            lo = at & 31;
            k = at >> 5;
          } else {
            int hi = 32;  // owner: the last lane whose offset is <= p
            lo = 0;
            while (hi - lo > 1) {
              const int mid = (lo + hi) >> 1;
              if (W.map[w].off[mid] <= p) lo = mid; else hi = mid;
            }
            k = p - W.map[w].off[lo];
          }
          PairSlot& ps = W.pairs[w][k][lo];
          const uint32_t j = ps.m;
          const float4 rr = W.ray[w][lo];
          const uint32_t src = W.src[w][lo];
          const Class32 c = classify32(objs[W.base[w][lo] + j], rr.x, rr.y, rr.z, rr.w, ps.key,
                                       (src >> 8) == j ? (int)(src & 0xffu) : -1);
          PairSlot o;
          o.key = c.key;
          o.ub = c.ub;
          o.s = c.s;
          o.m = j | ((uint32_t)(c.leaf + 1) << 16) | ((uint32_t)(c.face + 1) << 24);
          ps = o;
        }
        __syncwarp();
        for (int k = 0; k < cnt; ++k) {
          const PairSlot ps = W.pairs[w][k][lane];
          if (ps.ub < INFINITY) thr = fminf(thr, ps.ub * (1.0f + 1e-4f) + 1e-4f);
          if (!(ps.key <= thr)) continue;
          if (nc == CAND) {  // full: drop candidates the bound has since excluded
            int wr = 0;
            for (int q2 = 0; q2 < CAND; ++q2)
              if (W.cand[w][q2][lane].key <= thr) W.cand[w][wr++][lane] = W.cand[w][q2][lane];
            nc = wr;
          }
          if (nc < CAND) W.cand[w][nc++][lane] = ps;
          else overflow = true;
        }
        __syncwarp();
      };
      const GridRec& G = grid_of<MULTI>(S, pass_scene);
      const uint32_t gnx = CULL ? G.nx : 0u;
      if (gnx == 0) {
        // every object in table order
        for (uint32_t j0 = g_lo; j0 < g_hi; j0 += SCAN_CHUNK) {
          const uint32_t jn = min((uint32_t)SCAN_CHUNK, g_hi - j0);
          int cnt = 0;
          if (mine) my_tests += jn;
          for (uint32_t jj = 0; jj < jn; ++jj) {
            const uint32_t j = j0 + jj;
            const float4 h = MULTI ? __ldg(&S.bounds[j]) : *reinterpret_cast<const float4*>(&objs[j]);
            float lb;
            if (mine && bound_test(h, ox, oy, dx, dy, thr, lb)) {
              PairSlot& ps = W.pairs[w][cnt++][lane];
              ps.key = lb;
              ps.m = j - g_lo;  // scene-local object index
            }
          }
          classify_fold(cnt);
        }
      } else {
        // Culled: every lane walks the cells its own ray crosses, nearest first, and stops
        // at the first cell entered beyond its bound thr.  The walk moves one cell in x or
        // in y at a time, so the cells of an object's range that it visits are consecutive:
        // an object whose range holds the previous cell was tested there and is skipped,
        // and each object is tested at most once per ray.  A list entry carries a bit for each
        // side on which the object's range goes on (CELL_*); the one of the side the walk came
        // from says that the previous cell held the object.
        const uint32_t gny = G.ny;
        const float gx0 = G.x0, gy0 = G.y0, cw = G.cw, ch = G.ch, margin = G.margin;
        const uint32_t* cstart = S.cell_start + G.cell_base;
        const uint32_t* cobj = S.cell_obj + G.list_base;
        // (approximate: the grid's margin is some thousand ulp of its coordinates)
        const float idx = fabsf(dx) > 1e-30f ? __fdividef(1.0f, dx) : 0.0f;
        const float idy = fabsf(dy) > 1e-30f ? __fdividef(1.0f, dy) : 0.0f;
        const int sx = dx > 0.0f ? 1 : -1, sy = dy > 0.0f ? 1 : -1;
        int ix = 0, iy = 0;
        uint32_t came = 0;  // CELL_* bit of the side the walk entered the cell by (0: first cell)
        float tx = INFINITY, ty = INFINITY;
        uint32_t p = 0, pe = 0, steps = 0;
        bool act = mine, linear = false;
        if (act) {
          if (!(fabsf(ox) + fabsf(oy) <= G.reach)) {
            // an origin this far out carries FP32 errors above the margin: every object
            linear = true;
            pe = g_hi - g_lo;
          } else {
            const float bx1 = gx0 + (float)gnx * cw, by1 = gy0 + (float)gny * ch;
            float t0 = 0.0f, t1 = INFINITY;
            if (idx != 0.0f) {
              const float a = (gx0 - ox) * idx, b = (bx1 - ox) * idx;
              t0 = fmaxf(t0, fminf(a, b));
              t1 = fminf(t1, fmaxf(a, b));
            } else if (!(ox >= gx0 && ox <= bx1)) {
              t1 = -1.0f;
            }
            if (idy != 0.0f) {
              const float a = (gy0 - oy) * idy, b = (by1 - oy) * idy;
              t0 = fmaxf(t0, fminf(a, b));
              t1 = fminf(t1, fmaxf(a, b));
            } else if (!(oy >= gy0 && oy <= by1)) {
              t1 = -1.0f;
            }
            act = t0 <= t1 && t0 <= thr + margin;
            if (act) {
              const float fx = fminf(fmaxf(floorf((ox + dx * t0 - gx0) * G.iw), 0.0f), (float)(gnx - 1));
              const float fy = fminf(fmaxf(floorf((oy + dy * t0 - gy0) * G.ih), 0.0f), (float)(gny - 1));
              ix = (int)fx;
              iy = (int)fy;
              tx = idx != 0.0f ? (gx0 + (float)(ix + (dx > 0.0f ? 1 : 0)) * cw - ox) * idx : INFINITY;
              ty = idy != 0.0f ? (gy0 + (float)(iy + (dy > 0.0f ? 1 : 0)) * ch - oy) * idy : INFINITY;
              const uint32_t c = (uint32_t)iy * gnx + (uint32_t)ix;
              p = __ldg(cstart + c);
              pe = __ldg(cstart + c + 1);
            }
          }
        }
        // tests the object of a list entry with bound h, unless met in the previous cell
        auto test = [&](uint32_t e, const float4& h, int& cnt) {
          if (e & came) return;
          ++my_tests;
          float lb;
          if (bound_test(h, ox, oy, dx, dy, thr, lb)) {
            PairSlot& ps = W.pairs[w][cnt++][lane];
            ps.key = lb;
            ps.m = e & CELL_OBJ;
          }
        };
        while (__any_sync(0xffffffffu, act)) {
          // The lanes test the objects of their cells side by side, then those without pairs step
          // to their next cells; a lane with pairs waits for the fold (a hit in its cell may end
          // its walk there), and the warp folds after WALK_CELLS steps at the latest.
          int cnt = 0;
          for (int st = 0;; ++st) {
            while (__any_sync(0xffffffffu, act && p < pe && cnt + 2 <= SCAN_CHUNK)) {
              if (act && p < pe && cnt + 2 <= SCAN_CHUNK) {
                const bool two = p + 1 < pe;
                const uint32_t e0 = linear ? p : __ldg(cobj + p);
                const uint32_t e1 = two ? (linear ? p + 1 : __ldg(cobj + p + 1)) : e0;
                p += two ? 2u : 1u;
                const uint32_t j0 = e0 & CELL_OBJ, j1 = e1 & CELL_OBJ;
                const float4 h0 = MULTI ? __ldg(&S.bounds[g_lo + j0]) : *reinterpret_cast<const float4*>(&objs[j0]);
                const float4 h1 = MULTI ? __ldg(&S.bounds[g_lo + j1]) : *reinterpret_cast<const float4*>(&objs[j1]);
                test(e0, h0, cnt);
                if (two) test(e1, h1, cnt);
              }
            }
            const bool step = act && p >= pe && (cnt == 0 || linear);
            if (st == WALK_CELLS || !__any_sync(0xffffffffu, step)) break;
            if (!step) continue;
            if (linear || ++steps > gnx + gny + 2) {
              act = false;
              continue;
            }
            float te;  // the next cell along the ray
            if (tx <= ty) {
              ix += sx;
              te = tx;
              tx = (gx0 + (float)(ix + (sx > 0 ? 1 : 0)) * cw - ox) * idx;
              came = sx > 0 ? CELL_LEFT : CELL_RIGHT;
            } else {
              iy += sy;
              te = ty;
              ty = (gy0 + (float)(iy + (sy > 0 ? 1 : 0)) * ch - oy) * idy;
              came = sy > 0 ? CELL_BELOW : CELL_ABOVE;
            }
            if (ix < 0 || iy < 0 || ix >= (int)gnx || iy >= (int)gny || !(te <= thr + margin) || te == INFINITY) {
              act = false;
            } else {
              const uint32_t c = (uint32_t)iy * gnx + (uint32_t)ix;
              p = __ldg(cstart + c);
              pe = __ldg(cstart + c + 1);
            }
          }
          classify_fold(cnt);
        }
      }
    }
    // the ray record again (primaries were stored above): the scan does not keep it live
    if (valid) r = q[idx];
    const SceneLoc slp = scene_of<MULTI>(S, valid ? r.scene : 0u);
    bool emit = false;
    float x1 = 0.0f, y1 = 0.0f;
    uint8_t eflags = 0;
    if (valid) {
      ScanRec sc;
      sc.nc = 0;
      sc.overflow = overflow ? 1 : 0;
      sc.leaf = -1;
      sc.face = -1;
      sc.t32 = 0.0f;
      sc.s32 = 0.0f;
      sc.thr = thr;
      int list = -1;
      if (dead) {
        sc.nc = NC_DEAD;
      } else {
        int m = 0;
        PairSlot first;
        first.key = INFINITY;
        for (int k = 0; k < nc; ++k) {
          const PairSlot ps = W.cand[w][k][lane];
          if (!(ps.key <= thr)) continue;
          if (m == 0) first = ps;
          sc.cand[m++] = (uint16_t)(ps.m & 0xffffu);
        }
        sc.nc = (uint8_t)m;
        const int leaf = (int)((first.m >> 16) & 0xffu) - 1, face = (int)(first.m >> 24) - 1;
        if (!overflow && m == 1 && first.key == first.ub && leaf >= 0) {
          // a single candidate whose nearest root is certain: only that root is refined
          const uint32_t oinfo = reinterpret_cast<const uint32_t*>(&objs[slp.base + sc.cand[0]])[3];
          const int kind = leaf_kind_of(oinfo, leaf);
          sc.leaf = (int8_t)leaf;
          sc.face = (int8_t)face;
          sc.t32 = first.ub;
          sc.s32 = first.s;
          list = kind == LEAF_CIRCLE ? LIST_REFINE_CIRCLE : kind == LEAF_RECT ? LIST_REFINE_RECT
               : kind == LEAF_SEGMENT ? LIST_REFINE_SEGMENT : LIST_REFINE_CUBIC;
        } else if (m > 0 || overflow) {
          list = LIST_FULL;
        } else {
          // no object can be hit: leave through the canvas (tracer.rs:482-488)
          float L;
          if (!EXACT && fast_canvas_exit(slp.aspect, r, x1, y1, L)) {
            emit = true;
            ++my_visits;
            eflags = r.flags | (near_cutoff(r.c, slp.cutoff) ? LG_PATH_NEAR_DEGENERATE : 0) |
                     (L > ILL_COND ? LG_PATH_ILL_CONDITIONED : 0);
          } else {
            list = LIST_EXIT;
          }
        }
      }
      B.scan[idx] = sc;
      list_append(B, gen, list, (uint32_t)idx);
    }
    emit_segments(S, B, emit, r, x1, y1, eflags, -1, my_near, my_ill);
  }
  __syncwarp();
  const uint32_t my_cls = lane_id() == 0 ? cls_count[w] : 0u;
  if (EXACT)  // every visit is counted by the bounce
    add_block_counts<2>({my_tests, my_cls}, {&B.ctr->bound_tests, &B.ctr->object_tests});
  else
    add_block_counts<5>({my_tests, my_cls, my_visits, my_near, my_ill},
                        {&B.ctr->bound_tests, &B.ctr->object_tests, &B.ctr->visits, &B.ctr->near, &B.ctr->ill});
}

template __global__ void k_scan<false, false, false, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<false, false, true, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<false, true, false, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<false, true, true, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, false, false, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, false, true, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, true, false, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, true, true, 8>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<false, false, false, 16>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<false, false, true, 16>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<false, true, false, 16>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<false, true, true, 16>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, false, false, 16>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, false, true, 16>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, true, false, 16>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_scan<true, true, true, 16>(SceneDev, TraceBufs, uint32_t, int);

__device__ __forceinline__ void store_hit(HitRec& o, int obj, const Hit64& h, float ev, uint8_t flags) {
  o.obj = obj < 0 ? HIT_NONE : (uint16_t)obj;
  o.t = h.t; o.px = h.px; o.py = h.py; o.nx = h.nx; o.ny = h.ny;
  o.k = h.k;
  o.leaf = h.leaf;
  o.ev = ev;
  o.flags = flags;
}

// One launch refines the four leaf-kind lists one after the other (a warp's rays come from
// one list except at the seams, so the kinds stay apart as in four launches).
template <bool MULTI>
__global__ void __launch_bounds__(256) k_refine(SceneDev S, TraceBufs B, uint32_t gen) {
  stamp_start(B.ctr, gen, 1);
  auto count = [&](int l) -> uint64_t {
    const unsigned long long c = B.ctr->list_count[gen][l];
    return c < B.queue_cap ? c : B.queue_cap;
  };
  const uint64_t o1 = count(LIST_REFINE_CIRCLE), o2 = o1 + count(LIST_REFINE_RECT);
  const uint64_t o3 = o2 + count(LIST_REFINE_SEGMENT), n = o3 + count(LIST_REFINE_CUBIC);
  const RayRec* q = B.queue[gen & 1];
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t idx = i < o1 ? B.list[LIST_REFINE_CIRCLE][i]
                       : i < o2 ? B.list[LIST_REFINE_RECT][i - o1]
                       : i < o3 ? B.list[LIST_REFINE_SEGMENT][i - o2] : B.list[LIST_REFINE_CUBIC][i - o3];
    const RayRec r = q[idx];
    const ScanRec sc = B.scan[idx];
    Hit64 h;
    if (refine_root(S, obj_base_of<MULTI>(S, r.scene) + sc.cand[0], sc.leaf, sc.face, sc.t32, sc.s32, r.ox, r.oy,
                    r.dx, r.dy, h)) {
      store_hit(B.hit[idx], sc.cand[0], h, INFINITY, 0);
    } else {  // cannot refine (degenerate): solve it fully after this kernel
      B.scan[idx].leaf = LEAF_REFINE_FAILED;
      const unsigned long long slot = atomicAdd(&B.ctr->list_count[gen][LIST_FULL], 1ull);
      if (slot < B.queue_cap) B.list[LIST_FULL][slot] = idx;
    }
  }
}

template __global__ void k_refine<false>(SceneDev, TraceBufs, uint32_t);
template __global__ void k_refine<true>(SceneDev, TraceBufs, uint32_t);

template <bool MULTI>
__global__ void __launch_bounds__(256, 2) k_full(SceneDev S, TraceBufs B, uint32_t gen, int smem_fits) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  unsigned long long n = B.ctr->list_count[gen][LIST_FULL];
  if (n > B.queue_cap) n = B.queue_cap;
  if ((uint64_t)blockIdx.x * blockDim.x >= n) return;  // no ray for this CTA
  bool failed;
  const ObjScan* objs = stage_objects(S, reinterpret_cast<ObjScan*>(smem_raw), &bar, !MULTI && smem_fits != 0, B.ctr,
                                      failed);
  if (failed) return;
  const RayRec* q = B.queue[gen & 1];
  uint32_t my_solves = 0;
  // block-uniform loop: the CTA's warps solve one class at a time together (a barrier
  // between classes), so that one solver's code is in flight per CTA
  for (uint64_t base = blockIdx.x * (uint64_t)blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = base + threadIdx.x;
    const bool valid = i < n;
    const uint32_t idx = B.list[LIST_FULL][valid ? i : base];  // idle lanes read a real entry, store nothing
    const RayRec r = q[idx];
    const ScanRec sc = B.scan[idx];
    const SceneLoc sl = scene_of<MULTI>(S, r.scene);
    const ObjScan* sobjs = objs + sl.base;
    df best_d2 = DF_INF, second = DF_INF;
    Near ev{INFINITY, ray_tol(r.ex, r.ea)};
    int best = -1;
    Hit64 bh;
    bh.leaf = 0;
    // the nearest hit is the minimum of (d2, object index): candidates may be solved in
    // any order, so the warp runs one solve class at a time
    auto consider = [&](uint32_t j) {
      Hit64 hh;
      df d2;
      ++my_solves;
      if (obj_solve64(S, sl.base + j, r.ox, r.oy, r.dx, r.dy, hh, d2, ev)) {
        if (d2 < best_d2 || (d2 == best_d2 && (int)j < best)) {
          second = best_d2;
          best_d2 = d2;
          best = (int)j;
          bh = hh;
        } else if (d2 < second) {
          second = d2;
        }
      }
    };
    {
      uint32_t pending = valid && !sc.overflow ? (1u << sc.nc) - 1u : 0u;
      uint32_t cls[CAND];
      for (int k = 0; k < CAND; ++k)
        cls[k] = k < sc.nc ? solve_class(reinterpret_cast<const uint32_t*>(&sobjs[sc.cand[k]])[3]) : 7u;
      for (uint32_t c = 0; c < N_SOLVE_CLASSES; ++c) {
        for (;;) {
          int k = -1;
          for (int kk = 0; kk < CAND; ++kk)
            if (k < 0 && ((pending >> kk) & 1u) && cls[kk] == c) k = kk;
          if (!__any_sync(0xffffffffu, k >= 0)) break;
          if (k >= 0) {
            pending &= ~(1u << k);
            consider(sc.cand[k]);
          }
        }
        __syncthreads();
      }
    }
    if (!valid) continue;
    if (sc.overflow) {  // list overflow (rare): every object that passes the FP32 filters, in order
      const float ox = r.ox.hi, oy = r.oy.hi, dx = r.dx.hi, dy = r.dy.hi;
      for (uint32_t j = 0; j < sl.n; ++j) {
        const float4 h = *reinterpret_cast<const float4*>(&sobjs[j]);
        float lb;
        if (!bound_test(h, ox, oy, dx, dy, sc.thr, lb)) continue;
        if (!(classify32(sobjs[j], ox, oy, dx, dy, lb, j == r.src_obj ? (int)r.src_leaf : -1).key <= sc.thr)) continue;
        consider(j);
      }
    }
    uint8_t fl = sc.overflow ? LG_PATH_FALLBACK : 0;
    // a tie between two objects, within the band or within what the ray's error bound moves d2
    if (best >= 0 && second.hi < INFINITY &&
        (second - best_d2).hi <= fmaxf(1e-10f * best_d2.hi, 4.0f * sqrtf(best_d2.hi) * ev.tol))
      fl |= LG_PATH_NEAR_DEGENERATE;
    store_hit(B.hit[idx], best, bh, ev.ev, fl);
  }
  add_block_counts<1>({my_solves}, {&B.ctr->fp64_solves});
}
template __global__ void k_full<false>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_full<true>(SceneDev, TraceBufs, uint32_t, int);

// What a ray visit leaves: its segment, and up to two rays that start at (ox, oy): the reflected
// (or mirrored) one with direction d0 and colour scaled by f0, and the refracted one.
struct Bounce {
  bool emit, child0, child1;
  float x1, y1;
  int hit;
  uint8_t flags, cflags, leaf;  // of the segment, of the children; leaf the children start on
  uint16_t medium1;             // of the refracted ray
  float f0, f1, ex0, ea0, ex1, ea1;
  df ox, oy, dx0, dy0, dx1, dy1;
};

template <bool MULTI, bool CULL>
__device__ __forceinline__ void bounce(const SceneDev& S, const ObjScan* objs, const RayRec& r, const ScanRec& sc,
                                       const HitRec* hrec, Bounce& v) {
  v.emit = v.child0 = v.child1 = false;
  const SceneLoc sl = scene_of<MULTI>(S, r.scene);
  uint8_t fl = r.flags;
  if (near_cutoff(r.c, sl.cutoff)) fl |= LG_PATH_NEAR_DEGENERATE;
  const df ox = r.ox, oy = r.oy, dx = r.dx, dy = r.dy;
  HitRec bh;
  bh.obj = HIT_NONE;
  bh.flags = 0;
  bh.ev = INFINITY;
  if (sc.nc > 0) bh = *hrec;
  fl |= bh.flags;
  const int best = bh.obj == HIT_NONE ? -1 : (int)bh.obj;
  if (best >= 0 ? bh.ev <= bh.t.hi * (1.0f + 1e-6f) + 1e-12f : bh.ev < INFINITY) fl |= LG_PATH_NEAR_DEGENERATE;

  if (best >= 0) {
    const ObjInfo oi = S.info[sl.base + best];
    v.emit = true;
    v.x1 = bh.px.hi; v.y1 = bh.py.hi;
    v.hit = best;
    // first-order error at the hit: lateral offset L, offset along the surface ds
    const df ddn = dx * bh.nx + dy * bh.ny;
    const float ci_abs = fabsf(ddn.hi);
    const float kap = fminf(bh.k, 1e30f);
    // The FP64 quadratic of a curved surface (b^2 - a c with |b| ~ |o - c|) moves the
    // reference's own hit by about eps64 |o - c|^2 / (r cos) along the ray: an origin far
    // from a small circle makes the reference's result itself uncertain, and the path is
    // flagged once that, carried through the bounces, passes ILL_COND.
    const float oc = bh.t.hi + (kap > 0.0f ? 1.0f / kap : 0.0f);
    const float ref_solve = kap > 0.0f ? FP64_SOLVE_EPS * oc * oc * kap / fmaxf(ci_abs, 1e-6f) : 0.0f;
    const float L = r.ex + bh.t.hi * r.ea + DF_ROUND * (1.0f + fabsf(bh.px.hi) + fabsf(bh.py.hi)) + ref_solve;
    const float ds = L / fmaxf(ci_abs, 1e-6f);
    if (L > ILL_COND) fl |= LG_PATH_ILL_CONDITIONED;
    if (oi.flags & INFO_MATERIAL) {
      // medium on the far side (tracer.rs:428-442); "origin inside obj" at the midpoint
      df n2 = DF_ONE;
      uint16_t m2 = MEDIUM_AIR;
      bool near = false;
      // membership behind an FP32 pre-test whose band covers the ray's error bound: a decided point
      // lies outside the precise test's near-degenerate band too
      auto inside = [&](uint32_t k, df x, df y) -> bool {
        const int m = obj_member32(MULTI ? S.scan[k] : objs[k], x.hi, y.hi, 1e-6f + L);
        return m >= 0 ? m == 1 : obj_contains64(S, k, x, y, near, L);
      };
      if (inside(sl.base + (uint32_t)best, DF_HALF * (ox + bh.px), DF_HALF * (oy + bh.py))) {
        const float px32 = bh.px.hi, py32 = bh.py.hi;
        // the first other material object, in table order, that contains the hit point
        auto far_side = [&](uint32_t k) -> bool {
          if ((int)k == best) return false;
          const float4 h = MULTI ? __ldg(&S.bounds[sl.base + k]) : *reinterpret_cast<const float4*>(&objs[sl.base + k]);
          if (!(__float_as_uint(h.w) & INFO_MATERIAL)) return false;
          const float ex = px32 - h.x, ey = py32 - h.y;
          const float tol = 2e-6f * (fabsf(px32) + fabsf(py32) + fabsf(h.x) + fabsf(h.y) + h.z) + 1e-6f;
          if (ex * ex + ey * ey > (h.z + tol) * (h.z + tol)) return false;
          if (!inside(sl.base + k, bh.px, bh.py)) return false;
          n2 = S.info[sl.base + k].n;
          m2 = (uint16_t)k;
          return true;
        };
        const GridRec& G = grid_of<MULTI>(S, r.scene);
        if (!CULL || G.nx == 0) {
          for (uint32_t k = 0; k < sl.n; ++k)
            if (far_side(k)) break;
        } else {
          // the hit point's cell lists, in table order, every object whose box holds it
          const float fx = fminf(fmaxf(floorf((px32 - G.x0) * G.iw), 0.0f), (float)(G.nx - 1));
          const float fy = fminf(fmaxf(floorf((py32 - G.y0) * G.ih), 0.0f), (float)(G.ny - 1));
          const uint32_t c = (uint32_t)fy * G.nx + (uint32_t)fx;
          const uint32_t* cs = S.cell_start + G.cell_base;
          const uint32_t* co = S.cell_obj + G.list_base;
          for (uint32_t q = __ldg(cs + c), qe = __ldg(cs + c + 1); q < qe; ++q)
            if (far_side(__ldg(co + q) & CELL_OBJ)) break;
        }
      } else {
        n2 = oi.n;
        m2 = (uint16_t)best;
      }
      if (near) fl |= LG_PATH_NEAR_DEGENERATE;
      // Ray::refract: Snell + unpolarised Fresnel, TIR -> reflectance 1
      df nx = bh.nx, ny = bh.ny;
      df ci = -ddn;
      if (df_neg(ci)) { ci = -ci; nx = -nx; ny = -ny; }
      const df n1 = r.medium == MEDIUM_AIR ? DF_ONE
                    : r.medium == MEDIUM_LIGHT ? S.lights[sl.light_base + r.light].n0 : S.info[sl.base + r.medium].n;
      const df eta = n1 / n2;
      const df k = DF_ONE - eta * eta * (DF_ONE - ci * ci);
      if (fabsf(k.hi) <= 1e-10f) fl |= LG_PATH_NEAR_DEGENERATE;
      float R = 1.0f;
      bool refr = false;
      df tx = DF_ZERO, ty = DF_ZERO, ct = DF_ZERO;
      if (!df_neg(k)) {
        ct = dsqrt(k);
        const df m = eta * ci - ct;
        tx = eta * dx + m * nx;
        ty = eta * dy + m * ny;
        refr = true;
        const df dsn = n1 * ci + n2 * ct, dp = n1 * ct + n2 * ci;
        if (dsn.hi != 0.0f && dp.hi != 0.0f) {
          const df rs = (n1 * ci - n2 * ct) / dsn, rp = (n1 * ct - n2 * ci) / dp;
          R = (DF_HALF * (rs * rs + rp * rp)).hi;
        }
      }
      v.flags = fl | (refr ? 0 : LG_PATH_TIR);
      v.f0 = R;
      v.f1 = 1.0f - R;
      const df ci2 = ci * 2.0f;
      v.dx0 = dx + ci2 * nx;
      v.dy0 = dy + ci2 * ny;
      v.dx1 = tx;
      v.dy1 = ty;
      v.medium1 = m2;
      const float gain = eta.hi * ci.hi / fmaxf(ct.hi, 1e-6f);
      v.ex1 = ds * ct.hi + L;
      v.ea1 = gain * (r.ea + kap * ds) + kap * ds;
      v.child0 = true;
      v.child1 = refr;
    } else {
      v.flags = fl;
      const df dn2 = ddn * 2.0f;  // Ray::reflect: the colour as it is
      v.dx0 = dx - dn2 * bh.nx;
      v.dy0 = dy - dn2 * bh.ny;
      v.f0 = 1.0f;
      v.child0 = true;
    }
    v.ox = bh.px;
    v.oy = bh.py;
    v.ex0 = L;
    v.ea0 = r.ea + 2.0f * kap * ds;
    v.leaf = bh.leaf;
    v.cflags = fl;
  } else {
    // canvas exit: nearest hit with the canvas rectangle (tracer.rs:482-488)
    Leaf64 canvas;
    canvas.kind = LEAF_RECT;
    canvas.p[0] = DF_ZERO; canvas.p[1] = DF_ZERO; canvas.p[2] = DF_ONE; canvas.p[3] = DF_ZERO;
    canvas.p[4] = sl.aspect; canvas.p[5] = DF_ONE;
    Hit64 ch[3];
    Near cev{INFINITY, ray_tol(r.ex, r.ea)};
    const int nh = leaf_hits64(canvas, ox, oy, dx, dy, ch, cev);
    if (nh > 0) {
      int bi = 0;
      for (int q = 1; q < nh; ++q)
        if (ch[q].t < ch[bi].t) bi = q;
      v.emit = true;
      v.x1 = ch[bi].px.hi; v.y1 = ch[bi].py.hi;
      v.hit = -1;
      const float L = r.ex + ch[bi].t.hi * r.ea;
      v.flags = fl | (cev.ev < INFINITY ? LG_PATH_NEAR_DEGENERATE : 0) | (L > ILL_COND ? LG_PATH_ILL_CONDITIONED : 0);
    }
  }
  // children: the next generation skips colours below the cutoff (tracer.rs:378-384)
  const bool deeper = (uint32_t)r.gen + 1 < sl.max_bounce;
  const float k0[4] = {__fmul_rn(r.c[0], v.f0), __fmul_rn(r.c[1], v.f0), __fmul_rn(r.c[2], v.f0), r.c[3]};
  const float k1[4] = {__fmul_rn(r.c[0], v.f1), __fmul_rn(r.c[1], v.f1), __fmul_rn(r.c[2], v.f1), r.c[3]};
  v.child0 = v.child0 && deeper && !below_cutoff(k0, sl.cutoff);
  v.child1 = v.child1 && deeper && !below_cutoff(k1, sl.cutoff);
}

__device__ __forceinline__ uint4 bits2(df a, df b) {
  return make_uint4(__float_as_uint(a.hi), __float_as_uint(a.lo), __float_as_uint(b.hi), __float_as_uint(b.lo));
}
__device__ __forceinline__ ChildRay child_df(const RayRec& r, const Bounce& v, df dx, df dy, float f, float ex, float ea,
                                             const float* cutoff, uint64_t path, uint16_t medium) {
  ChildRay c{{bits2(v.ox, v.oy), bits2(dx, dy)}, {__fmul_rn(r.c[0], f), __fmul_rn(r.c[1], f), __fmul_rn(r.c[2], f)},
             ex, ea, path, v.cflags, v.leaf, medium, (uint16_t)v.hit};
  const float k[4] = {c.c[0], c.c[1], c.c[2], r.c[3]};
  if (near_cutoff(k, cutoff)) c.flags |= LG_PATH_NEAR_DEGENERATE;
  if (!(ex <= ILL_COND && ea <= ILL_COND)) c.flags |= LG_PATH_ILL_CONDITIONED;
  return c;
}

template <bool MULTI, bool CULL>
__global__ void __launch_bounds__(256, 3) k_bounce(SceneDev S, TraceBufs B, uint32_t gen, int smem_fits) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  stamp_start(B.ctr, gen, 2);
  // the rays with work: every work list of this generation, one after the other
  uint64_t off[N_LISTS + 1];
  off[0] = 0;
  for (int l = 0; l < N_LISTS; ++l) {
    const unsigned long long c = B.ctr->list_count[gen][l];
    off[l + 1] = off[l] + (c < B.queue_cap ? c : B.queue_cap);
  }
  const uint64_t total = off[N_LISTS];
  if ((uint64_t)blockIdx.x * blockDim.x >= total) return;  // no ray for this CTA
  bool failed;
  const ObjScan* objs = stage_objects(S, reinterpret_cast<ObjScan*>(smem_raw), &bar, !MULTI && smem_fits != 0, B.ctr,
                                      failed);
  if (failed) return;
  const RayRec* qin = B.queue[gen & 1];
  RayRec* qout = B.queue[(gen + 1) & 1];
  const unsigned lane = lane_id();
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  uint32_t my_visits = 0, my_near = 0, my_ill = 0;
  for (uint64_t base = warp * 32; base < total; base += nwarps * 32) {
    const uint64_t i = base + lane;
    Bounce v;
    v.emit = v.child0 = v.child1 = false;
    v.flags = 0;
    v.hit = -1;
    v.f0 = v.f1 = 1.0f;
    RayRec r;
    if (i < total) {
      int l = 0;
      while (i >= off[l + 1]) ++l;
      const uint32_t idx = B.list[l][i - off[l]];
      const ScanRec sc = B.scan[idx];
      if (!(l < LIST_FULL && sc.leaf == LEAF_REFINE_FAILED)) {  // those are in the full list too
        r = qin[idx];
        ++my_visits;
        bounce<MULTI, CULL>(S, objs, r, sc, &B.hit[idx], v);
      }
    }
    unsigned long long seg, s0, s1;
    reserve_out(B, gen, v.emit, v.child0, v.child1, seg, s0, s1);
    if (v.emit) store_segment(S, B, r, v.x1, v.y1, v.flags, v.hit, seg, my_near, my_ill);
    if (v.child0 || v.child1) {
      const SceneLoc sl = scene_of<MULTI>(S, r.scene);
      if (v.child0 && s0 < B.queue_cap)
        store_child(qout + s0, r, child_df(r, v, v.dx0, v.dy0, v.f0, v.ex0, v.ea0, sl.cutoff, r.path, r.medium));
      if (v.child1 && s1 < B.queue_cap)
        store_child(qout + s1, r, child_df(r, v, v.dx1, v.dy1, v.f1, v.ex1, v.ea1, sl.cutoff, r.path | (1ull << r.gen), v.medium1));
    }
  }
  stamp_end(B.ctr, gen);
  add_block_counts<3>({my_visits, my_near, my_ill}, {&B.ctr->visits, &B.ctr->near, &B.ctr->ill});
}
template __global__ void k_bounce<false, false>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_bounce<false, true>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_bounce<true, false>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_bounce<true, true>(SceneDev, TraceBufs, uint32_t, int);

// ------------------------------------------------------------------- visiting order
// Generations > 0: a counting sort of the queue entries by scene, place and direction (keys and
// histogram, exclusive scan, scatter of entry indices).  Rays that start in one cell of the canvas
// in one octant of directions walk the same grid cells to the same few objects, so that a warp's
// lanes stay together in the scan's walk and leaf code, and through the work lists in the solve, the
// bounce and the segments' bins.  Bound by memory: the keys read a sector pair of each 80-byte entry.
__device__ __forceinline__ unsigned long long warp_scene_atomic(unsigned* slot_base, uint32_t s, bool on) {
  const unsigned act = __activemask();
  const unsigned grp = __match_any_sync(act, on ? s : 0xffffffffu);
  if (!on) return 0;
  const int leader = __ffs(grp) - 1;
  unsigned base = 0;
  if ((int)lane_id() == leader) base = atomicAdd(&slot_base[s], (unsigned)__popc(grp));
  base = __shfl_sync(grp, base, leader);
  return base + __popc(grp & lanemask_lt());
}

// queued rays per scene
__global__ void k_scene_hist(SceneDev S, TraceBufs B, uint32_t gen, unsigned* count) {
  const uint64_t n = n_real_of(S, B, gen);
  const RayRec* q = B.queue[gen & 1];
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t s = q[i].scene;
    warp_scene_atomic(count, s, s < S.n_scenes);
  }
}

// The lowest `bits` bits (0, or 3 + 2 k: an octant of directions and 2^k x 2^k cells of the
// canvas; a start outside it counts to the nearest cell).  Any value serves: it only orders.
__device__ __forceinline__ uint32_t place_key(float ox, float oy, float dx, float dy, float aspect, uint32_t bits) {
  if (bits < 3) return 0;
  const uint32_t k = (bits - 3) >> 1;
  const int n = 1 << k;
  const int cx = min(max((int)((ox / aspect + 1.0f) * (0.5f * (float)n)), 0), n - 1);
  const int cy = min(max((int)((oy + 1.0f) * (0.5f * (float)n)), 0), n - 1);
  const uint32_t oct = (dx > 0.0f ? 1u : 0u) | (dy > 0.0f ? 2u : 0u) | (fabsf(dx) > fabsf(dy) ? 4u : 0u);
  return (uint32_t)((cy << k) + cx) * 8u + oct;
}

// A double's value as a float, truncated (on the integer pipe: a conversion would issue on the
// FP64 pipe); beyond FP32's range or NaN some large value, below it zero.
__device__ __forceinline__ float rough(uint32_t hi) {
  const int e = (int)((hi >> 20) & 0x7ffu) - 896;
  const uint32_t m = e <= 0 ? 0u : e >= 255 ? 0x7f000000u : ((uint32_t)e << 23) | ((hi & 0xfffffu) << 3);
  return __uint_as_float((hi & 0x80000000u) | m);
}

template <bool MULTI, bool EXACT>
__global__ void k_sort_keys(SceneDev S, TraceBufs B, uint32_t gen, uint32_t bits, uint32_t* keys, unsigned* count) {
  const uint64_t n = n_real_of(S, B, gen);
  if (!sorts<MULTI>(n)) return;
  const RayRec* q = B.queue[gen & 1];
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint4 o = reinterpret_cast<const uint4*>(q + i)[0], d = reinterpret_cast<const uint4*>(q + i)[1];
    const uint32_t s = MULTI ? q[i].scene : 0u;
    const bool on = s < S.n_scenes;
    // the leading part of a double-float, or of a double
    auto lead = [](uint32_t lo, uint32_t hi) { return EXACT ? rough(hi) : __uint_as_float(lo); };
    uint32_t key = 0;
    if (on)
      key = (s << bits) + place_key(lead(o.x, o.y), lead(o.z, o.w), lead(d.x, d.y), lead(d.z, d.w),
                                    scene_of<MULTI>(S, s).aspect.hi, bits);
    keys[i] = on ? key : 0xffffffffu;
    warp_scene_atomic(count, key, on);
  }
}
template __global__ void k_sort_keys<false, false>(SceneDev, TraceBufs, uint32_t, uint32_t, uint32_t*, unsigned*);
template __global__ void k_sort_keys<false, true>(SceneDev, TraceBufs, uint32_t, uint32_t, uint32_t*, unsigned*);
template __global__ void k_sort_keys<true, false>(SceneDev, TraceBufs, uint32_t, uint32_t, uint32_t*, unsigned*);
template __global__ void k_sort_keys<true, true>(SceneDev, TraceBufs, uint32_t, uint32_t, uint32_t*, unsigned*);

// off = exclusive scan of count, 16384 bins a CTA; both hold a multiple of 16 bins.  A CTA sums the
// bins before its own itself: eight CTAs read 1.8 MB of L2 in all, where one CTA that walked 2^17
// bins took 47 us a generation (a 64-scene batch 73.1 -> 72.3 ms).  (Done by the last CTA of
// k_sort_keys instead, the fences and the larger CTAs cost more than the launch.)
template <bool MULTI>
__global__ void __launch_bounds__(1024) k_sort_offsets(SceneDev S, TraceBufs B, uint32_t gen, const unsigned* count,
                                                       unsigned* off, uint32_t n_bins) {
  if (!sorts<MULTI>(n_real_of(S, B, gen))) return;
  __shared__ unsigned wsum[32], wbefore[32];
  const unsigned lane = lane_id(), wid = threadIdx.x >> 5;
  const uint32_t first = blockIdx.x * SORT_CTA_BINS, i = first + 16 * threadIdx.x;
  unsigned before = 0;
  for (uint32_t j = 4 * threadIdx.x; j < first; j += 4 * blockDim.x) {
    const uint4 v = *reinterpret_cast<const uint4*>(count + j);
    before += v.x + v.y + v.z + v.w;
  }
  uint4 c[4] = {};
  if (i < n_bins)
    for (int k = 0; k < 4; ++k) c[k] = reinterpret_cast<const uint4*>(count + i)[k];
  unsigned sum = 0;
  for (int k = 0; k < 4; ++k) sum += c[k].x + c[k].y + c[k].z + c[k].w;
  before = __reduce_add_sync(0xffffffffu, before);
  unsigned incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
    if ((int)lane >= o) incl += y;
  }
  if (lane == 31) wsum[wid] = incl;
  if (lane == 0) wbefore[wid] = before;
  __syncthreads();
  const unsigned w = wsum[lane];
  unsigned at = __reduce_add_sync(0xffffffffu, wbefore[lane] + (lane < wid ? w : 0u)) + incl - sum;
  if (i >= n_bins) return;
  for (int k = 0; k < 4; ++k) {
    uint4 v;
    v.x = at; at += c[k].x;
    v.y = at; at += c[k].y;
    v.z = at; at += c[k].z;
    v.w = at; at += c[k].w;
    reinterpret_cast<uint4*>(off + i)[k] = v;
  }
}
template __global__ void k_sort_offsets<false>(SceneDev, TraceBufs, uint32_t, const unsigned*, unsigned*, uint32_t);
template __global__ void k_sort_offsets<true>(SceneDev, TraceBufs, uint32_t, const unsigned*, unsigned*, uint32_t);

// the entries' indices in sorted order; clears the histogram for the next generation
template <bool MULTI>
__global__ void k_sort_scatter(SceneDev S, TraceBufs B, uint32_t gen, const uint32_t* keys, unsigned* off, uint32_t* order,
                               unsigned* count, uint32_t n_bins) {
  const uint64_t n = n_real_of(S, B, gen);
  if (!sorts<MULTI>(n)) return;
  for (uint32_t i = 4 * (blockIdx.x * blockDim.x + threadIdx.x); i < n_bins; i += 4 * gridDim.x * blockDim.x)
    *reinterpret_cast<uint4*>(count + i) = make_uint4(0u, 0u, 0u, 0u);
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t key = keys[i];
    const bool on = key != 0xffffffffu;
    const unsigned long long pos = warp_scene_atomic(off, key, on);
    if (on && pos < n) order[pos] = (uint32_t)i;
  }
}
template __global__ void k_sort_scatter<false>(SceneDev, TraceBufs, uint32_t, const uint32_t*, unsigned*, uint32_t*,
                                               unsigned*, uint32_t);
template __global__ void k_sort_scatter<true>(SceneDev, TraceBufs, uint32_t, const uint32_t*, unsigned*, uint32_t*,
                                              unsigned*, uint32_t);

// ------------------------------------------------------------------- overlays
// A point of the string-mod curve (string_mod.rs:33-85), the same FP64 operations as the
// oracle: angle (turns * n) * 2 pi / m, the library's own sine and cosine.
__device__ void string_mod_point(const lg_string_mod& sm, uint64_t n, double& x, double& y) {
  using namespace lgx;
  const uint64_t k = sm.turns * n;
  if (sm.curve == LG_CURVE_COMPLEX_EXP) {
    // (re + i im)^(u32)k by binary powering (num-complex 0.4.6, Pow<u32> for &Complex)
    uint32_t e = (uint32_t)k;
    if (e == 0) { x = 1.0; y = 0.0; return; }
    double br = sm.curve_f[0], bi = sm.curve_f[1];
    while ((e & 1u) == 0) {
      const double r = sub(mul(br, br), mul(bi, bi)), i = add(mul(br, bi), mul(bi, br));
      br = r; bi = i; e >>= 1;
    }
    double ar = br, ai = bi;
    while (e > 1) {
      e >>= 1;
      const double r = sub(mul(br, br), mul(bi, bi)), i = add(mul(br, bi), mul(bi, br));
      br = r; bi = i;
      if (e & 1u) {
        const double r2 = sub(mul(ar, br), mul(ai, bi)), i2 = add(mul(ar, bi), mul(ai, br));
        ar = r2; ai = i2;
      }
    }
    x = ar; y = ai;
    return;
  }
  const double angle = dvd(mul((double)k, 2.0 * 3.141592653589793), (double)sm.modulo);
  double s, c;
  if (sm.curve == LG_CURVE_HYPOTROCHOID) {
    const double r = (double)sm.curve_u[0], big = (double)sm.curve_u[1], d = (double)sm.curve_u[2];
    const double smr = sub(big, r), ratio = add(smr, d);
    double s2, c2;
    sincos_x(angle, s, c);
    sincos_x(dvd(mul(angle, smr), r), s2, c2);
    x = dvd(add(mul(smr, c), mul(d, c2)), ratio);
    y = dvd(sub(mul(smr, s), mul(d, s2)), ratio);
  } else if (sm.curve == LG_CURVE_LISSAJOUS) {
    double s2, c2;
    sincos_x(add(mul((double)sm.curve_u[0], angle), sm.curve_f[0]), s, c);
    sincos_x(mul((double)sm.curve_u[1], angle), s2, c2);
    x = s;
    y = s2;
  } else {
    sincos_x(angle, s, c);
    x = c;
    y = s;
  }
}

// The point that line iix of a string mod joins to point iix, by the mod's mode
// (string_mod.rs:112-117; u64 arithmetic wrapping like Rust's release build).
__device__ __forceinline__ uint64_t string_mod_target(const lg_string_mod& sm, uint64_t iix) {
  const uint64_t m = sm.modulo;
  if (sm.mode == LG_SM_ADD) return (iix + sm.num) % m;
  if (sm.mode == LG_SM_MUL) return (iix * sm.num) % m;
  uint64_t b = sm.mode == LG_SM_POW ? iix : sm.num, e = sm.mode == LG_SM_POW ? (uint32_t)sm.num : (uint32_t)iix, p = 1;
  while (e) {
    if (e & 1) p *= b;
    b *= b;
    e >>= 1;
  }
  return p % m;
}

// StringMod::get_color (string_mod.rs:124-150): the f32 mean of the matching modulo colours,
// summed in table order, else the base colour.
__device__ void string_mod_color(const lg_string_mod& sm, const lg_mod_color* colors, uint32_t n_colors,
                                 uint64_t ix, float* out) {
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  uint32_t cnt = 0;
  for (uint32_t k = 0; k < n_colors; ++k) {
    const lg_mod_color& e = colors[k];
    if (ix % e.modulo == e.rem) {
#pragma unroll
      for (int ch = 0; ch < 4; ++ch) acc[ch] = __fadd_rn(acc[ch], e.color[ch]);
      ++cnt;
    }
  }
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) out[ch] = cnt ? __fdiv_rn(acc[ch], (float)cnt) : sm.color[ch];
}

// Overlays drawn after the trace: the control polygons of curved mirrors (tracer.rs:341-346)
// appended to the segment ring, and the string-mod lines (string_mod.rs:104-122) written to
// their own table, one per point: chord iix joins point iix and point ix(iix) of the mode,
// each vertex with its own colour.
__global__ void k_overlay(SceneDev S, TraceBufs B, const uint32_t* cubic_objs, const uint16_t* cubic_scene,
                          uint32_t n_cubic, lg_string_mod sm, ChordArgs CA) {
  const uint64_t n_ctrl = 3ull * n_cubic;
  const uint64_t total = n_ctrl + sm.modulo;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    if (i < n_ctrl) {
      lg_segment s;
      lg_path_record pr;
      pr.path = 0; pr.light = 0xffff; pr.flags = 0; pr.hit = -1;
      uint16_t scene = 0;
      if (cubic_scene) scene = cubic_scene[i / 3];
      const uint32_t k = cubic_objs[i / 3];
      const int q = (int)(i % 3);
      const Leaf64& L = S.leaves[S.info[k].leaf_begin];
      s.x0 = L.p[2 * q].hi; s.y0 = L.p[2 * q + 1].hi;
      s.x1 = L.p[2 * q + 2].hi; s.y1 = L.p[2 * q + 3].hi;
      s.color[0] = 1.f; s.color[1] = 0.f; s.color[2] = 0.f; s.color[3] = 1.f;
      pr.primary = k; pr.gen = (uint8_t)q; pr.source = LG_SRC_CONTROL_LINE;
      const unsigned long long slot = atomicAdd(&B.ctr->seg_count, 1ull);
      if (slot < B.seg_cap) {
        B.segs[slot] = s;
        if (B.seg_scene) B.seg_scene[slot] = scene;
        if (S.record_paths) B.paths[slot] = pr;
      }
    } else {
      const uint64_t m = sm.modulo, iix = i - n_ctrl;
      const uint64_t ix = string_mod_target(sm, iix);
      double xa, ya, xb, yb;
      if (CA.pts) {  // nested: points iix and ix of the outer mod's crossings (string_mod.rs:118-119)
        const double2 pa = CA.pts[iix % CA.n_pts], pb = CA.pts[ix % CA.n_pts];
        xa = pa.x; ya = pa.y; xb = pb.x; yb = pb.y;
      } else {
        string_mod_point(sm, iix % m, xa, ya);
        string_mod_point(sm, ix % m, xb, yb);
      }
      lg_chord c;
      c.x0 = (float)xa; c.y0 = (float)ya; c.x1 = (float)xb; c.y1 = (float)yb;
      string_mod_color(sm, CA.colors, CA.n_colors, iix, c.color0);
      string_mod_color(sm, CA.colors, CA.n_colors, ix, c.color1);
      if (CA.out) CA.out[iix] = c;
    }
  }
}

// ---------------------------------------------------------- nested string mods
// StringMod::line_crossings_as_points (string_mod.rs:87-102): line k of the outer mod joins
// point k and point ix(k) of its curve, in FP64 (pts[2k], pts[2k + 1]) and rounded to FP32; a thread
// per point.
__global__ void k_sm_lines(lg_string_mod sm, double2* pts, float2* pts32) {
  const uint64_t m = sm.modulo;
  for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < 2 * m; e += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = e >> 1;
    double x, y;
    string_mod_point(sm, ((e & 1) ? string_mod_target(sm, k) : k) % m, x, y);
    pts[e] = make_double2(x, y);
    pts32[e] = make_float2((float)x, (float)y);
  }
}

// Crossing of segments ab and cd (collision2d's LineSegment::intersect is not vendored; this
// is the definition include/lg.h states): the 2x2 parametric solve a + t (b - a) =
// c + u (d - c), each FP64 operation rounded on its own, a crossing when the determinant is
// not zero and t, u lie in [0, 1]; the point is a + t (b - a).
__device__ __noinline__ bool seg_cross_x(double2 a, double2 b, double2 c, double2 d, double2& p) {
  using namespace lgx;
  const double rx = sub(b.x, a.x), ry = sub(b.y, a.y), sx = sub(d.x, c.x), sy = sub(d.y, c.y);
  const double den = sub(mul(rx, sy), mul(ry, sx));
  if (den == 0.0) return false;
  const double wx = sub(c.x, a.x), wy = sub(c.y, a.y);
  const double t = dvd(sub(mul(wx, sy), mul(wy, sx)), den);
  const double u = dvd(sub(mul(wx, ry), mul(wy, rx)), den);
  if (!(t >= 0.0 && t <= 1.0 && u >= 0.0 && u <= 1.0)) return false;
  p.x = add(a.x, mul(rx, t));
  p.y = add(a.y, mul(ry, t));
  return true;
}

// Whether a pair crosses, in FP32 where that is certain: 1 yes, 0 no, -1 undecided.  Coordinates
// rounded to FP32 and the products' roundings move the determinant and the numerators by at
// most 4e-7 times the products of the sums of magnitudes (some 3 2^-24 each); with the sign of the
// determinant taken out, t and u lie in [0, 1] where 0 <= numerator <= |determinant|.
__device__ __forceinline__ int seg_cross32(float4 ab, float4 cd) {
  const float rx = ab.z - ab.x, ry = ab.w - ab.y, sx = cd.z - cd.x, sy = cd.w - cd.y;
  const float ma = fabsf(ab.x) + fabsf(ab.y) + fabsf(ab.z) + fabsf(ab.w);
  const float mc = fabsf(cd.x) + fabsf(cd.y) + fabsf(cd.z) + fabsf(cd.w);
  const float e = 1e-6f * (ma + mc) * (ma + mc) + 1e-30f;
  const float den = rx * sy - ry * sx, wx = cd.x - ab.x, wy = cd.y - ab.y;
  const float D = fabsf(den), sg = den < 0.0f ? -1.0f : 1.0f;
  const float T = sg * (wx * sy - wy * sx), U = sg * (wx * ry - wy * rx);
  if (!(D > e) || !(ma + mc < 1e18f)) return -1;  // (no product overflows below 1e18)
  if (T < -e || T > D + 2.0f * e || U < -e || U > D + 2.0f * e) return 0;
  return T > e && T < D - 2.0f * e && U > e && U < D - 2.0f * e ? 1 : -1;
}

// pair q of m (m - 1), in the reference's order: diff = q / m + 1 (outer loop), line a = q % m
// joined with line b = (a + diff) % m
struct CrossPair {
  uint32_t a, b;
};
__device__ __forceinline__ CrossPair cross_pair(uint32_t m, uint32_t q) {
  const uint32_t diff = q / m, a = q - diff * m, b = a + diff + 1;
  return CrossPair{a, b >= m ? b - m : b};
}

// Bound: the FP32 tests of m (m - 1) pairs.  A warp takes 32 consecutive pairs and leaves a mask of
// those that cross; FP64 decides only pairs within the FP32 rounding.  (All in FP64, with 64-bit
// index divisions and both quotients, 1.4 M pairs took 133 us here and 276 us again in the write.)
__global__ void __launch_bounds__(CROSS_THREADS) k_cross_count(const double2* pts, const float4* lines32, uint32_t m,
                                                               uint32_t* blk, uint32_t* masks) {
  __shared__ uint32_t warp_sums[CROSS_WARPS];
  const uint32_t n_pairs = m * (m - 1), w = threadIdx.x >> 5;
  uint32_t count = 0;
  for (int row = 0; row < CROSS_ROWS; ++row) {
    const uint32_t q = blockIdx.x * CROSS_PAIRS_PER_BLOCK + row * CROSS_THREADS + threadIdx.x;
    bool on = false;
    if (q < n_pairs) {
      const CrossPair P = cross_pair(m, q);
      const int k = seg_cross32(__ldg(lines32 + P.a), __ldg(lines32 + P.b));
      double2 p;
      on = k > 0 || (k < 0 && seg_cross_x(pts[2 * P.a], pts[2 * P.a + 1], pts[2 * P.b], pts[2 * P.b + 1], p));
    }
    const uint32_t mask = __ballot_sync(0xffffffffu, on);
    if (lane_id() == 0) masks[blockIdx.x * CROSS_MASKS + row * CROSS_WARPS + w] = mask;
    count += __popc(mask);
  }
  if (lane_id() == 0) warp_sums[w] = count;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t all = 0;
    for (int k = 0; k < CROSS_WARPS; ++k) all += warp_sums[k];
    blk[blockIdx.x] = all;
  }
}

// one CTA of 1024 threads: exclusive scan of the per-block counts in place
__global__ void __launch_bounds__(1024) k_cross_scan(uint32_t* blk, uint32_t n_blk, unsigned long long* total) {
  __shared__ unsigned long long carry;
  __shared__ uint32_t warp_sums[32];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const unsigned lane = lane_id(), w = threadIdx.x >> 5;
  for (uint32_t base = 0; base < n_blk; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < n_blk ? blk[i] : 0u;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)lane >= o) incl += y;
    }
    if (lane == 31) warp_sums[w] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (unsigned k = 0; k < blockDim.x / 32; ++k) {
      if (k < w) before += warp_sums[k];
      all += warp_sums[k];
    }
    const unsigned long long c0 = carry;
    if (i < n_blk) blk[i] = (uint32_t)(c0 + before + incl - v);
    __syncthreads();
    if (threadIdx.x == 0) carry = c0 + all;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// The crossing points in pair order: the block's offset, the masks before this one, the lane's
// place in its mask.
__global__ void __launch_bounds__(CROSS_THREADS) k_cross_write(const double2* pts, uint32_t m, const uint32_t* blk_off,
                                                                const uint32_t* masks, double2* out) {
  __shared__ uint32_t off[CROSS_MASKS + 1];
  __shared__ uint16_t list[CROSS_PAIRS_PER_BLOCK];
  const uint32_t w = threadIdx.x >> 5;
  static_assert(CROSS_MASKS == 128, "four masks per lane of one warp");
  if (threadIdx.x < 32) {  // exclusive sums of the block's 128 mask counts
    const uint4 v = reinterpret_cast<const uint4*>(masks + blockIdx.x * CROSS_MASKS)[threadIdx.x];
    const uint32_t c[4] = {(uint32_t)__popc(v.x), (uint32_t)__popc(v.y), (uint32_t)__popc(v.z), (uint32_t)__popc(v.w)};
    const uint32_t own = c[0] + c[1] + c[2] + c[3];
    uint32_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)threadIdx.x >= o) incl += y;
    }
    uint32_t at = incl - own;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      off[4 * threadIdx.x + k] = at;
      at += c[k];
    }
    if (threadIdx.x == 31) off[CROSS_MASKS] = at;
  }
  __syncthreads();
  // the block's crossing pairs side by side, so that the FP64 work fills its warps
  for (int row = 0; row < CROSS_ROWS; ++row) {
    const uint32_t k = row * CROSS_WARPS + w, mask = masks[blockIdx.x * CROSS_MASKS + k];
    if ((mask >> lane_id()) & 1u) list[off[k] + __popc(mask & lanemask_lt())] = (uint16_t)(row * CROSS_THREADS + threadIdx.x);
  }
  __syncthreads();
  const uint64_t base = blk_off[blockIdx.x];
  for (uint32_t i = threadIdx.x; i < off[CROSS_MASKS]; i += CROSS_THREADS) {
    using namespace lgx;
    const CrossPair P = cross_pair(m, blockIdx.x * CROSS_PAIRS_PER_BLOCK + list[i]);
    const double2 a = pts[2 * P.a], b = pts[2 * P.a + 1], c = pts[2 * P.b], d = pts[2 * P.b + 1];
    const double rx = sub(b.x, a.x), ry = sub(b.y, a.y), sx = sub(d.x, c.x), sy = sub(d.y, c.y);
    const double t = dvd(sub(mul(sub(c.x, a.x), sy), mul(sub(c.y, a.y), sx)), sub(mul(rx, sy), mul(ry, sx)));
    out[base + i] = make_double2(add(a.x, mul(rx, t)), add(a.y, mul(ry, t)));
  }
}

}  // namespace lgd
