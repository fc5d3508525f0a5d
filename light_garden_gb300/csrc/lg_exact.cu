// lg_exact.cu — the solve and bounce kernels of the exact FP64 precision mode.
//
// In LG_PRECISION_EXACT one generation is k_scan (FP32 search, lg_trace.cu: candidates of
// the nearest hit, in work lists) -> k_solve_x -> k_bounce_x.  Both kernels here evaluate
// the restated collision2d formulas of lg_x64.cuh in IEEE double with every operation
// rounded on its own, so every decision of Tracer::trace (tracer.rs:360-493: nearest hit
// with strict < in object order, medium rule, refract / reflect, colour split, canvas exit)
// is taken on the same FP64 values a CPU evaluation of those formulas computes, and the
// segments and child rays come out bit for bit equal.
//
// Rays and hits keep their FP64 coordinates in the 8-byte df slots of RayRec / HitRec (xd /
// xdf move the bits).
#include "lg_kernels.cuh"
#include "lg_trace_common.cuh"

// CTAs per SM the exact kernels' registers are sized for (build-time, for sweeps)
#ifndef LG_SOLVE_X_BLOCKS
#define LG_SOLVE_X_BLOCKS 4
#endif
#ifndef LG_BOUNCE_X_BLOCKS
#define LG_BOUNCE_X_BLOCKS 3
#endif

namespace lgd {

using lgx::V;

__device__ __forceinline__ V ray_o(const RayRec& r) { return lgx::mk(xd(r.ox), xd(r.oy)); }
__device__ __forceinline__ V ray_d(const RayRec& r) { return lgx::mk(xd(r.dx), xd(r.dy)); }

// Membership of object k (object.rs:240-253): mirrors enclose nothing.
__device__ __forceinline__ bool obj_contains_x(const SceneDev& S, uint32_t k, V p, uint32_t* fl) {
  const ObjInfo& oi = S.info[k];
  if (oi.flags & INFO_NO_CONTAINS) return false;
  return lgx::object_contains_tree(S.xgeo, S.xnode + oi.xnode_begin, (int)oi.xnode_count, p, fl);
}

// obj_contains_x behind the FP32 pre-test (k scene-global).
__device__ __forceinline__ bool obj_contains_f(const SceneDev& S, uint32_t k, V p, uint32_t* fl) {
  const int m = obj_member32(S.scan[k], (float)p.x, (float)p.y, 1e-6f);
  if (m >= 0) return m == 1;
  return obj_contains_x(S, k, p, fl);
}

// Light start media (tracer.rs:280-287: the last object with a material containing the
// light's position) and spot base angles (light.rs:230-234), once per frame.  Bound: latency
// (a chain of dependent loads and FP64 tests per object).  A warp per light tests 32 objects at
// a time from the end of the table, each in FP32 first; one thread per light walking the table
// took 1.2 ms on 256 CSG objects and 3.6 ms on a batch with a 1024-object scene.
template <bool MULTI>
__global__ void k_light_setup_x(SceneDev S) {
  const uint32_t l0 = S.serve ? S.light_lo : 0u, l1 = S.serve ? S.light_hi : S.n_lights;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t l = l0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); l < l1; l += warps) {
    LightDev& L = S.lights[l];
    const SceneLoc sl = scene_of<MULTI>(S, L.scene);
    const V p = lgx::mk(L.ox, L.oy);
    const uint32_t k = last_object_of_warp(sl.base, sl.n, [&](uint32_t j) {
      return (S.info[j].flags & INFO_MATERIAL) && obj_contains_f(S, j, p, nullptr);
    });
    if (lane_id() == 0) {
      L.n0x = k == 0xffffffffu ? 1.0 : S.info[k].n64;
      L.n0 = k == 0xffffffffu ? DF_ONE : S.info[k].n;
      L.dir_angle = lgx::spot_base_angle(L.vx, L.vy);
    }
  }
}
template __global__ void k_light_setup_x<false>(SceneDev);
template __global__ void k_light_setup_x<true>(SceneDev);

// ------------------------------------------------------------------ nearest hit
// Exact hit record in HitRec's slots: t, p, n as FP64, the event parameter ev in (k, ev).
__device__ __forceinline__ void store_hit_x(HitRec& o, int obj, const lgx::Hit& h, V n, int leaf, double ev,
                                            uint8_t flags) {
  o.obj = obj < 0 ? HIT_NONE : (uint16_t)obj;
  o.t = xdf(h.t); o.px = xdf(h.p.x); o.py = xdf(h.p.y); o.nx = xdf(n.x); o.ny = xdf(n.y);
  const df e = xdf(ev);
  o.k = e.hi;
  o.ev = e.lo;
  o.leaf = (uint8_t)leaf;
  o.flags = flags;
}

// Nearest hit of object k (scene-global index) with the ray: the minimum distance_squared
// over the object's hits, the first one on ties (tracer.rs:412-424 per object).  Returns
// that distance (INFINITY: no hit).  Out of line, so the solve kernel keeps one copy of the
// geometry code and its own registers for the ray state.
static __device__ __noinline__ double obj_best_x(const SceneDev& S, uint32_t k, V o, V d, double& ev, lgx::Hit& best) {
  const ObjInfo& oi = S.info[k];
  double ob = INFINITY;
  lgx::object_hits(S.xgeo, S.xnode + oi.xnode_begin, (int)oi.xnode_count, o, d, ev, [&](const lgx::Hit& h) {
    const V dv = lgx::vsub(h.p, o);
    const double d2 = lgx::dot(dv, dv);
    if (lgx::plt(d2, ob)) {
      ob = d2;
      best = h;
    }
  });
  return ob;
}

// The FP64 hit of an object whose nearest root the FP32 scan proved (a single candidate with a
// certain root and, for a two-leaf CSG object, certain membership of that root's point in the
// other leaf): the very operations of object_hits, leaf_hits and object_normal for that root
// only, since the other roots, the other leaf and the membership tests cannot change which hit
// object_hits keeps.  side: the proved leaf; t32: its root; face: the rect face as 2 axis + (outward
// sign > 0); s32: a cubic's curve parameter.  A circle computes the quotient of its proved
// root (q / a or c / q, told apart by their FP32 values) and not the other; a rect the slab
// quotient of its proved face and not the other three; a segment its ray parameter and not the
// place along it; a cubic searches only the bracket that holds s32, and in it only near s32.
// False: no such hit (the caller solves the object whole).
__device__ __forceinline__ bool solve_proved_x(const SolveRec& G, V o, V d, int side, int face, float t32, float s32,
                                               double& t, V& p, V& n) {
  using namespace lgx;
  const uint32_t kind = G.kind;
  const bool two = (kind & 0xfu) == SR_TWO;
  // 16-byte loads: the record is gathered per lane, and every load is a trip of the texture pipe
  const double2* G2 = reinterpret_cast<const double2*>(&G);
  double2 org2 = make_double2(0.0, 0.0), rot2 = make_double2(1.0, 0.0);
  if (two) {
    org2 = __ldg(G2);
    rot2 = __ldg(G2 + 1);
    o = irot(vsub(o, mk(org2.x, org2.y)), rot2.x, rot2.y);
    d = irot(d, rot2.x, rot2.y);
  } else if (side != 0) {
    return false;
  }
  const V org = mk(org2.x, org2.y);
  const double2* L2 = G2 + (side ? 5 : 2);
  const double2 l0 = __ldg(L2), l1 = __ldg(L2 + 1);
  const uint32_t k = (side ? kind >> 8 : kind >> 4) & 0xfu;
  if (k == LEAF_CIRCLE) {
    const V ctr = mk(l0.x, l0.y), oc = vsub(o, ctr);
    const double r = l1.x;
    const double a = dot(d, d), b = dot(oc, d), cc = sub(dot(oc, oc), mul(r, r));
    const double disc = sub(mul(b, b), mul(a, cc));
    if (is_neg(disc)) return false;
    const double sq = sqr(disc);
    const double q = -add(b, is_neg(b) ? -sq : sq);
    if (is_zero(q)) return false;
    const float ra = (float)q / (float)a, rc = (float)cc / (float)q;  // selection only
    const bool first = fabsf(ra - t32) <= fabsf(rc - t32);
    t = dvd(first ? q : cc, first ? a : q);
    p = vadd(o, vscl(d, t));
    n = vscl(vsub(p, ctr), l1.y);
  } else if (k == LEAF_RECT) {
    if (face < 0) return false;
    const int ax = face >> 1;
    const bool pos = (face & 1) != 0;
    // the face's axis of irot(o - centre) and irot(d) alone: x' = c x + s y, y' = -s x + c y
    const double2 half = __ldg(L2 + 2);
    const double c = l1.x, s = l1.y;
    const V rel = vsub(o, mk(l0.x, l0.y));
    const double kx = ax ? -s : c, ky = ax ? c : s;
    const double O = add(mul(kx, rel.x), mul(ky, rel.y)), D = add(mul(kx, d.x), mul(ky, d.y));
    if (is_zero(D)) return false;
    const double h = ax ? half.y : half.x;
    t = dvd(sub(pos ? h : -h, O), D);
    p = vadd(o, vscl(d, t));
    const double sg = pos ? 1.0 : -1.0;
    n = rot(ax == 0 ? mk(sg, 0.0) : mk(0.0, sg), c, s);
  } else if (k == LEAF_SEGMENT) {  // the crossing lies well inside the segment: t alone
    const double2 nl = __ldg(L2 + 2);
    const V A = mk(l0.x, l0.y), e = vsub(mk(l1.x, l1.y), A);
    const double den = cross(d, e);
    if (is_zero(den)) return false;
    t = dvd(cross(vsub(A, o), e), den);
    p = vadd(o, vscl(d, t));
    n = mk(nl.x, nl.y);
  } else {  // cubic
    // the bracket between the derivative's roots that holds the proved curve parameter s32:
    // hits_cubic's operations for that bracket only (a parameter within 1e-4 of a knot takes the
    // whole object)
    if (!(s32 > 0.0f)) return false;
    const double2 l2 = __ldg(L2 + 2), l3 = __ldg(L2 + 3);
    const Cubic K{mk(l0.x, l0.y), mk(l1.x, l1.y), mk(l2.x, l2.y), mk(l3.x, l3.y)};
    const double a[4] = {cross(d, vsub(K.c0, o)), cross(d, K.c1), cross(d, K.c2), cross(d, K.c3)};
    double kn[4];
    int nk = 0;
    kn[nk++] = 0.0;
    const double qa = mul(3.0, a[3]), qb = mul(2.0, a[2]), qc = a[1];
    if (qa != 0.0) {
      const double disc = sub(mul(qb, qb), mul(mul(4.0, qa), qc));
      if (disc >= 0.0) {
        const double sq = sqr(disc);
        const double q = mul(-0.5, add(qb, qb >= 0 ? sq : -sq));
        // a root that FP32 puts outside [0, 1] is no knot: 2 stands for it
        const float e1 = __fdividef((float)q, (float)qa), e2 = __fdividef((float)qc, (float)q);
        double r1 = e1 < -0.01f || e1 > 1.01f ? 2.0 : dvd(q, qa);
        double r2 = q != 0.0 ? (e2 < -0.01f || e2 > 1.01f ? 2.0 : dvd(qc, q)) : r1;
        if (r1 > r2) { const double x = r1; r1 = r2; r2 = x; }
        if (r1 > 0.0 && r1 < 1.0) kn[nk++] = r1;
        if (r2 > 0.0 && r2 < 1.0 && (nk == 1 || r2 != kn[1])) kn[nk++] = r2;
      }
    } else if (qb != 0.0) {
      const double r = dvd(-qc, qb);
      if (r > 0.0 && r < 1.0) kn[nk++] = r;
    }
    kn[nk++] = 1.0;
    double lo = -1.0, hi = -1.0;
    for (int i = 0; i + 1 < nk; ++i)
      if ((double)s32 > kn[i] + 1e-4 && (double)s32 < kn[i + 1] - 1e-4) { lo = kn[i]; hi = kn[i + 1]; }
    if (!(lo >= 0.0)) return false;
    // f at s32 -+ 1e-4: where both values are well above the rounding of f and their signs differ,
    // f (monotone between the knots) keeps those signs beyond these points, to the bracket's ends
    const double wlo = sub((double)s32, 1e-4), whi = add((double)s32, 1e-4);
    const double fa = poly3(a, wlo), fb = poly3(a, whi);
    const float sc = 1e-9f * (fabsf((float)a[0]) + fabsf((float)a[1]) + fabsf((float)a[2]) + fabsf((float)a[3]));
    if (is_neg(fa) == is_neg(fb) || !(fabsf((float)fa) > sc) || !(fabsf((float)fb) > sc)) return false;
    const double sr = cubic_root(a, lo, hi, fa, wlo, whi);
    t = dvd(dot(vsub(cubic_point(K, sr), o), d), dot(d, d));
    p = vadd(o, vscl(d, t));
    const V dB = cubic_tangent(K, sr);
    const double l = sqr(dot(dB, dB));
    n = l > 0.0 ? mk(dvd(-dB.y, l), dvd(dB.x, l)) : unit(mk(-d.y, d.x));
  }
  if (!gt_pos(t, T_MIN)) return false;
  if (two) {  // lifted out of the Logic frame
    p = vadd(org, rot(p, rot2.x, rot2.y));
    n = rot(n, rot2.x, rot2.y);
  }
  return true;
}

// The nearest hit of one ray over candidate objects, each solved whole as tracer.rs:412-424
// does: the minimum distance_squared over an object's hits, then over objects with ties kept
// by the lower object index.
struct Nearest {
  double best_d2 = INFINITY, second = INFINITY, ev = INFINITY;
  int best = -1;
  lgx::Hit h{0.0, {0.0, 0.0}, {0.0, 0.0}, 0, 0};
  __device__ __forceinline__ void consider(const SceneDev& S, uint32_t base, uint32_t j, V o, V d) {
    lgx::Hit oh;
    const double ob = obj_best_x(S, base + j, o, d, ev, oh);
    if (!lgx::plt(ob, INFINITY)) return;
    if (lgx::plt(ob, best_d2) || (lgx::bits(ob) == lgx::bits(best_d2) && (int)j < best)) {
      second = best_d2;
      best_d2 = ob;
      best = (int)j;
      h = oh;
    } else if (lgx::plt(ob, second)) {
      second = ob;
    }
  }
  // the hit record with the near-degenerate flags of tracer.rs's decisions: ties within the
  // band, decisions in the band before the hit; the normal of the winning hit only
  __device__ __forceinline__ void store(const SceneDev& S, uint32_t base, V d, uint8_t fl, HitRec& out) const {
    if (best >= 0 && lgx::plt(second, INFINITY) && lgx::sub(second, best_d2) <= lgx::mul(lgx::BAND, best_d2)) fl |= lgx::NEAR;
    if (lgx::plt(ev, INFINITY) && (best < 0 || ev <= lgx::add(lgx::mul(h.t, 1.0 + 1e-6), 1e-12))) fl |= lgx::NEAR;
    V n = lgx::mk(0.0, 0.0);
    int leaf = 0;
    if (best >= 0) {
      const lgx::XNode* nd = S.xnode + S.info[base + best].xnode_begin;
      n = lgx::object_normal(S.xgeo, nd, d, h);
      leaf = lgx::hit_leaf(S.xgeo, nd, h);
    }
    store_hit_x(out, best, h, n, leaf, ev, fl);
  }
};

// A ray of a refine list whose root is not of SolveRec's kinds or turned out not to be there:
// its one candidate solved whole.
static __device__ __noinline__ void solve_one_x(const SceneDev& S, uint32_t base, uint32_t j, V o, V d, HitRec& out) {
  Nearest N;
  N.consider(S, base, j, o, d);
  N.store(S, base, d, 0, out);
}

// Every ray with candidates.  First the refine lists (one candidate, its root proved; a list per
// leaf kind, so a warp's rays take one path), straight from the SolveRec; then the full-solve
// list, where the CTA's warps take the candidates one solve class (circle, rect, segment, cubic /
// deep CSG, two-leaf CSG) at a time, with a barrier between classes, so that one geometry code
// path is in flight per CTA.
template <bool MULTI>
__global__ void __launch_bounds__(256, LG_SOLVE_X_BLOCKS) k_solve_x(SceneDev S, TraceBufs B, uint32_t gen) {
  stamp_start(B.ctr, gen, 1);
  uint64_t off[LIST_FULL + 1];
  off[0] = 0;
  for (int l = 0; l < LIST_FULL; ++l) {
    const unsigned long long c = B.ctr->list_count[gen][l];
    off[l + 1] = off[l] + (c < B.queue_cap ? c : B.queue_cap);
  }
  const uint64_t proved = off[LIST_FULL];
  unsigned long long full = B.ctr->list_count[gen][LIST_FULL];
  if (full > B.queue_cap) full = B.queue_cap;
  const uint64_t first = blockIdx.x * (uint64_t)blockDim.x;
  if (first >= proved && (gridDim.x - 1 - blockIdx.x) * (uint64_t)blockDim.x >= full) return;  // no ray for this CTA
  const RayRec* q = B.queue[gen & 1];
  uint32_t my_solves = 0;
  for (uint64_t i = first + threadIdx.x; i < proved; i += (uint64_t)gridDim.x * blockDim.x) {
    int l = 0;
    while (i >= off[l + 1]) ++l;
    const uint32_t idx = B.list[l][i - off[l]];
    const double2* rp = reinterpret_cast<const double2*>(q + idx);  // ox, oy, dx, dy
    const double2 o2 = __ldcg(rp), d2 = __ldcg(rp + 1);
    const ScanRec* sp = B.scan + idx;
    const uint32_t j = sp->cand[0];
    const uint4 tail = __ldcg(reinterpret_cast<const uint4*>(sp) + 1);  // nc, overflow, leaf, face | t32 | thr | s32
    const int side = (int8_t)(tail.x >> 16), face = (int8_t)(tail.x >> 24);
    const uint32_t base = MULTI ? S.scenes[q[idx].scene].obj_base : 0u;
    const V o = lgx::mk(o2.x, o2.y), d = lgx::mk(d2.x, d2.y);
    const SolveRec& G = S.solve[base + j];
    double t;
    V p, n;
    ++my_solves;
    if ((G.kind & 0xfu) != SR_TREE &&
        solve_proved_x(G, o, d, side, face, __uint_as_float(tail.y), __uint_as_float(tail.w), t, p, n)) {
      double2* hp = reinterpret_cast<double2*>(B.hit + idx);  // HitRec in four 16-byte stores
      hp[0] = make_double2(t, p.x);
      hp[1] = make_double2(p.y, n.x);
      const uint2 ny = make_uint2((uint32_t)__double2loint(n.y), (uint32_t)__double2hiint(n.y));
      const df ev = xdf(INFINITY);
      reinterpret_cast<uint4*>(hp)[2] = make_uint4(ny.x, ny.y, __float_as_uint(ev.hi), __float_as_uint(ev.lo));
      reinterpret_cast<uint4*>(hp)[3] = make_uint4(j | ((uint32_t)side << 16), 0u, 0u, 0u);
    } else {
      solve_one_x(S, base, j, o, d, B.hit[idx]);
    }
  }
  // block-uniform loop (the class barrier needs every thread), from the last CTA on: in a small
  // generation the first CTAs have the proved rays
  for (uint64_t base = (gridDim.x - 1 - blockIdx.x) * (uint64_t)blockDim.x; base < full; base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = base + threadIdx.x;
    const bool valid = i < full;
    const uint32_t idx = valid ? B.list[LIST_FULL][i] : 0u;
    const RayRec& r = q[idx];
    const ScanRec sc = B.scan[idx];
    const SceneLoc sl = scene_of<MULTI>(S, valid ? r.scene : 0u);
    const V o = ray_o(r), d = ray_d(r);
    Nearest N;
    {
      uint32_t pending = valid && !sc.overflow ? (1u << sc.nc) - 1u : 0u;
      uint32_t cls[CAND];
      for (int k = 0; k < CAND; ++k)
        cls[k] = (pending >> k) & 1u ? solve_class(__ldg(&S.scan[sl.base + sc.cand[k]].info)) : 7u;
      for (uint32_t c = 0; c < N_SOLVE_CLASSES; ++c) {
        for (;;) {
          int k = -1;
          for (int kk = 0; kk < CAND; ++kk)
            if (k < 0 && ((pending >> kk) & 1u) && cls[kk] == c) k = kk;
          if (!__any_sync(0xffffffffu, k >= 0)) break;
          if (k >= 0) {
            pending &= ~(1u << k);
            ++my_solves;
            N.consider(S, sl.base, sc.cand[k], o, d);
          }
        }
        __syncthreads();
      }
    }
    if (!valid) continue;
    if (sc.overflow) {  // candidate list overflow (rare): every object that passes the FP32 filters
      const ObjScan* sobjs = S.scan + sl.base;
      const float ox = (float)o.x, oy = (float)o.y, dx = (float)d.x, dy = (float)d.y;
      for (uint32_t j = 0; j < sl.n; ++j) {
        const float4 h = *reinterpret_cast<const float4*>(&sobjs[j]);
        float lb;
        if (!bound_test(h, ox, oy, dx, dy, sc.thr, lb)) continue;
        if (!(classify32(sobjs[j], ox, oy, dx, dy, lb, j == r.src_obj ? (int)r.src_leaf : -1).key <= sc.thr)) continue;
        ++my_solves;
        N.consider(S, sl.base, j, o, d);
      }
    }
    N.store(S, sl.base, d, sc.overflow ? LG_PATH_FALLBACK : 0, B.hit[idx]);
  }
  add_block_counts<1>({my_solves}, {&B.ctr->fp64_solves});
}
template __global__ void k_solve_x<false>(SceneDev, TraceBufs, uint32_t);
template __global__ void k_solve_x<true>(SceneDev, TraceBufs, uint32_t);

// ------------------------------------------------------------------ bounce
// Primary number v of a frame (light.rs:103-115, 163-174, 225-249) as a queue entry.
__device__ __forceinline__ void primary_rec(const SceneDev& S, uint64_t v, RayRec& r) {
  uint32_t l = 0, hi = S.n_lights;
  while (hi - l > 1) {  // the last light whose first primary is <= v
    const uint32_t mid = (l + hi) >> 1;
    if (S.lights[mid].first <= v) l = mid; else hi = mid;
  }
  const LightDev& L = S.lights[l];
  const uint64_t i = S.ray_offset + (uint64_t)S.ray_stride * (v - L.first);
  double ox, oy, dx, dy;
  lgx::primary_ray_x(L.kind, L.ox, L.oy, L.vx, L.vy, L.spot_angle, L.dir_angle, (double)L.num_rays, i, ox, oy, dx, dy);
  r.ox = xdf(ox); r.oy = xdf(oy); r.dx = xdf(dx); r.dy = xdf(dy);
  r.medium = MEDIUM_LIGHT;
  r.src_obj = SRC_NONE;
  r.src_leaf = 0;
  for (int k = 0; k < 4; ++k) r.c[k] = L.color[k];
  r.path = 0;
  r.prim = (uint32_t)i;
  r.light = (uint16_t)l;
  r.gen = 0;
  r.flags = 0;
  r._pad = 0;
  r.scene = 0;
  r.ex = r.ea = 0.0f;
}

// What a ray visit leaves: its segment, and up to two rays that start at (ox, oy): the reflected
// (or mirrored) one with direction d0 and colour scaled by f0, and the refracted one.
struct BounceX {
  bool emit, child0, child1;
  float x0, y0, x1, y1;
  int hit;
  uint8_t flags, cflags, leaf;  // of the segment, of the children; leaf the children start on
  uint16_t medium1;             // of the refracted ray
  float f0, f1;
  V o, d0, d1;
};

// the bits of two FP64 coordinates, as the queue holds them
__device__ __forceinline__ uint4 bits2(V a) {
  return make_uint4((uint32_t)__double2loint(a.x), (uint32_t)__double2hiint(a.x), (uint32_t)__double2loint(a.y),
                    (uint32_t)__double2hiint(a.y));
}
__device__ __forceinline__ ChildRay child_x(const RayRec& r, const BounceX& v, V d, float f, uint64_t path, uint16_t medium) {
  return ChildRay{{bits2(v.o), bits2(d)}, {__fmul_rn(r.c[0], f), __fmul_rn(r.c[1], f), __fmul_rn(r.c[2], f)},
                  0.0f, 0.0f, path, v.cflags, v.leaf, medium, (uint16_t)v.hit};
}

// A non-negative double as double-float (relative error 2^-48; below 2^-60 it is 0, above 2^60
// infinite), on the integer pipe: a conversion each way would issue on the FP64 pipe.
__device__ __forceinline__ df df_of(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int e = ((hi >> 20) & 0x7ff) - 1023;
  if (e < -60 || e > 60) return df{e > 60 ? INFINITY : 0.0f, 0.0f};
  const float h = __int_as_float(((e + 127) << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)lo >> 29));
  const float l = __fmul_rn(__uint2float_rn((unsigned)lo & 0x1fffffffu), __int_as_float((e - 52 + 127) << 23));
  return fast_two_sum(h, l);
}
// a + b with an absolute error of 2^-47 (|a| + |b|) (operator+ keeps a relative one)
__device__ __forceinline__ df add_abs(df a, df b) {
  const df s = two_sum(a.hi, b.hi);
  return fast_two_sum(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}

// The unpolarised Fresnel reflectance rounded to FP32, which is all the colour split uses
// (tracer.rs:454), from double-float copies of the indices and cosines: false unless the FP32
// rounding of the FP64 formula's value is certain.  Every term n cos is within 2^-46 of itself,
// so rs and rp are within 2^-44 and R within 2^-43 (|rs| + |rp| + R), the FP64 formula's own
// rounding included; the bound below takes 2^-41.  A copy that df_of gave as 0 makes one term of either
// quotient 0 (a and d, b and c, a and c or b and d), so that both are 1 or -1 and the sum's high part is
// 1, whose zero mantissa is never certain; two such copies may give 0 / 0, and an infinite one NaN or
// the same, and NaN compares false.  So FP64 decides all of these.  (The refracted cosine is 0 or at least
// 2^-27, the root of a difference from 1: its conversion loses nothing.)  The test fails for about one
// visit in 10^4.  In FP64 the two quotients, four products and their sums are half of a bounce's FP64
// instructions.
// A reflectance below 2^-26 (matched indices: a ray that leaves an object into the medium it
// is already in) needs no exact value when dead says that the reflected colour is below the
// cutoff whatever it is: the refracted share 1 - R is 1.
__device__ __forceinline__ bool fresnel_f32(df n1, df n2, df ci, df ct, bool dead, float& R) {
  const df a = n1 * ci, b = n2 * ct, c = n1 * ct, d = n2 * ci;
  const df rs = add_abs(a, -b) / add_abs(a, b), rp = add_abs(c, -d) / add_abs(c, d);
  const df q = add_abs(rs * rs, rp * rp);
  const float hi = __fmul_rn(0.5f, q.hi), lo = __fmul_rn(0.5f, q.lo);
  const int hb = __float_as_int(hi);
  const float err = 4.5474735e-13f * (fabsf(rs.hi) + fabsf(rp.hi) + hi);  // 2^-41
  const float half = __int_as_float((hb & 0x7f800000) - (24 << 23));     // half an ulp of hi
  R = hi;
  if (dead && hi + err < 1.4901161e-08f) return true;
  return hi > 1e-20f && hi < 2.0f && (hb & 0x7fffff) != 0 && fabsf(lo) + err < half;
}

// Ray::refract restated (collision2d; called at tracer.rs:444-450): reflected direction,
// refracted direction unless total internal reflection, unpolarised Fresnel reflectance (as
// FP32).  eta = n1 / n2; dead: see fresnel_f32.
__device__ __forceinline__ bool refract_x(V d, V n, double n1, double n2, df n1f, df n2f, double eta, bool dead, V& refl,
                                          V& refr, float& R, uint32_t& fl) {
  using namespace lgx;
  double ci = -dot(d, n);
  if (is_neg(ci)) {
    ci = -ci;
    n = mk(-n.x, -n.y);
  }
  refl = vadd(d, vscl(n, mul(2.0, ci)));
  const double k = sub(1.0, mul(mul(eta, eta), sub(1.0, mul(ci, ci))));
  if (bits(fabs(k)) <= bits(BAND)) fl |= NEAR;
  if (is_neg(k)) {
    R = 1.0f;
    return false;
  }
  const double ct = sqr(k);
  refr = vadd(vscl(d, eta), vscl(n, sub(mul(eta, ci), ct)));
  if (fresnel_f32(n1f, n2f, df_of(ci), df_of(ct), dead, R)) return true;
  const double ds = add(mul(n1, ci), mul(n2, ct)), dp = add(mul(n1, ct), mul(n2, ci));
  if (ds == 0.0 || dp == 0.0) {
    R = 1.0f;
    return true;
  }
  const double rs = dvd(sub(mul(n1, ci), mul(n2, ct)), ds);
  const double rp = dvd(sub(mul(n1, ct), mul(n2, ci)), dp);
  R = (float)mul(0.5, add(mul(rs, rs), mul(rp, rp)));
  return true;
}

// The canvas exit of a ray whose origin lies strictly inside the canvas [-aspect, aspect] x
// [-1, 1] and whose exit is clear of the corners and of the origin: the same hit and flags as
// the slab test of the canvas rectangle (hits_rect), which needs the far face of each axis
// only: (sign(D) h - O) / D is the very quotient the slab test takes as its exit parameter.
// Returns false (nothing decided) when any of those conditions fails.
__device__ __forceinline__ bool canvas_exit_inside(V o, V d, double aspect, double& ev, lgx::Hit& first, int& nh) {
  using namespace lgx;
  const double h[2] = {aspect, 1.0};
  const double O[2] = {o.x, o.y}, D[2] = {d.x, d.y};
  double far[2];
  float nr[2];
  for (int ax = 0; ax < 2; ++ax) {
    if (is_zero(D[ax]) || !(fabs(O[ax]) < h[ax])) return false;
    far[ax] = dvd(sub(D[ax] > 0.0 ? h[ax] : -h[ax], O[ax]), D[ax]);
    // the near face's parameter, roughly: only needed to rule out a corner-entry event
    nr[ax] = ((float)(D[ax] > 0.0 ? -h[ax] : h[ax]) - (float)O[ax]) / (float)D[ax];
  }
  const double tf = far[1] < far[0] ? far[1] : far[0];
  if (!(tf >= 1e-9)) return false;
  // the slab test's events: a corner entry (the two near parameters within the band of each
  // other) and an exit within the T_MIN band; the corner graze |tf - tn| <= 1e-10 (|tn| + tf + 1)
  // cannot happen for tn < 0 <= 1e-9 <= tf
  const float tn_abs = fmaxf(fabsf(nr[0]), fabsf(nr[1]));
  if (!(fabsf(nr[0] - nr[1]) > 1e-6f * (tn_abs + (float)tf + 1.0f))) return false;
  lgx::tmin_band(tf, ev);
  if (gt_pos(tf, T_MIN)) {
    first = mkhit(tf, o, d, mk(0.0, 0.0), 0);
    nh = 1;
  }
  return true;
}

template <bool MULTI, bool CULL>
__device__ __forceinline__ void bounce_x(const SceneDev& S, const RayRec& r, const ScanRec& sc, const HitRec* hrec,
                                         BounceX& v) {
  using namespace lgx;
  v.emit = v.child0 = v.child1 = false;
  const SceneLoc sl = scene_of<MULTI>(S, r.scene);
  uint32_t fl = r.flags;
  if (near_cutoff(r.c, sl.cutoff)) fl |= NEAR;  // tracer.rs:378-384 in the band
  const V o = ray_o(r), d = ray_d(r);
  v.x0 = (float)o.x;
  v.y0 = (float)o.y;
  int best = -1;
  V bp = mk(0.0, 0.0), bn = mk(0.0, 0.0);
  uint8_t leaf = 0;
  if (sc.nc > 0 || sc.overflow) {
    const HitRec h = *hrec;
    fl |= h.flags;
    if (h.obj != HIT_NONE) {
      best = (int)h.obj;
      bp = mk(xd(h.px), xd(h.py));
      bn = mk(xd(h.nx), xd(h.ny));
      leaf = h.leaf;
    }
  }
  if (best >= 0) {
    const ObjInfo& oi = S.info[sl.base + best];
    v.emit = true;
    v.x1 = (float)bp.x;
    v.y1 = (float)bp.y;
    v.hit = best;
    if (oi.flags & INFO_MATERIAL) {
      // the medium on the far side (tracer.rs:428-442); "origin inside obj" at the midpoint
      double n2 = 1.0;
      uint16_t m2 = MEDIUM_AIR;
      const V mid = vscl(vadd(o, bp), 0.5);
      if (obj_contains_f(S, sl.base + (uint32_t)best, mid, &fl)) {
        // the first other object (in table order) that contains the hit point and has a material
        const float px32 = (float)bp.x, py32 = (float)bp.y;
        auto far_side = [&](uint32_t k) -> bool {
          if ((int)k == best) return false;
          const float4 h = MULTI ? __ldg(&S.bounds[sl.base + k]) : __ldg(reinterpret_cast<const float4*>(&S.scan[k]));
          if (__float_as_uint(h.w) & INFO_NO_CONTAINS) return false;
          const float ex = px32 - h.x, ey = py32 - h.y;
          const float tol = 2e-6f * (fabsf(px32) + fabsf(py32) + fabsf(h.x) + fabsf(h.y) + h.z) + 1e-6f;
          if (ex * ex + ey * ey > (h.z + tol) * (h.z + tol)) return false;  // far outside: no member, no band
          if (!obj_contains_f(S, sl.base + k, bp, &fl)) return false;
          if (!(__float_as_uint(h.w) & INFO_MATERIAL)) return false;
          n2 = S.info[sl.base + k].n64;
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
        n2 = oi.n64;
        m2 = (uint16_t)best;
      }
      // n1 / n2 without a division where one side is air: x / 1 = x, and 1 / n is in the table
      double n1 = 1.0, eta;
      df n1f = DF_ONE, n2f = DF_ONE;
      if (r.medium == MEDIUM_LIGHT) {
        const LightDev& L = S.lights[sl.light_base + r.light];
        n1 = L.n0x;
        n1f = L.n0;
      } else if (r.medium != MEDIUM_AIR) {
        const ObjInfo& mi = S.info[sl.base + r.medium];
        n1 = mi.n64;
        n1f = mi.n;
      }
      if (m2 != MEDIUM_AIR) n2f = S.info[sl.base + m2].n;
      if (bits(n2) == bits(1.0)) eta = n1;
      else if (bits(n1) == bits(1.0)) eta = S.info[sl.base + m2].inv_n64;
      else eta = dvd(n1, n2);
      V rl, rr = mk(0.0, 0.0);
      float refl;
      bool dead = true;  // c R <= c 2^-26 < cutoff in every channel
#pragma unroll
      for (int i = 0; i < 3; ++i) dead = dead && r.c[i] >= 0.0f && __fmul_rn(r.c[i], 1.4901161e-08f) < sl.cutoff[i];
      const bool refr = refract_x(d, bn, n1, n2, n1f, n2f, eta, dead, rl, rr, refl, fl);
      v.flags = (uint8_t)((fl & 0xffu) | (refr ? 0u : (uint32_t)LG_PATH_TIR));
      v.f0 = refl;
      v.f1 = __fsub_rn(1.0f, refl);
      v.d0 = rl;
      v.d1 = rr;
      v.medium1 = m2;
      v.child0 = true;
      v.child1 = refr;
    } else {  // Ray::reflect (tracer.rs:476-480): the colour as it is
      v.flags = (uint8_t)fl;
      const double dn = dot(d, bn);
      v.d0 = vsub(d, vscl(bn, mul(2.0, dn)));
      v.f0 = 1.0f;
      v.child0 = true;
    }
    v.o = bp;
    v.leaf = leaf;
    v.cflags = (uint8_t)fl;
  } else {
    // canvas exit (tracer.rs:482-488): nearest hit with the canvas rectangle
    const double aspect = MULTI ? S.scenes[r.scene].aspect64 : S.aspect64;
    double cev = INFINITY;
    int nh = 0;
    Hit first{INFINITY, mk(0.0, 0.0), mk(0.0, 0.0), 0, 0};
    if (!canvas_exit_inside(o, d, aspect, cev, first, nh)) {
      lg_geo canvas;
      canvas.kind = LG_GEO_RECT;
      canvas.origin[0] = 0.0; canvas.origin[1] = 0.0;
      canvas.rot[0] = 1.0; canvas.rot[1] = 0.0;
      canvas.v[2] = aspect;  // half width and height
      canvas.v[3] = 1.0;
      hits_rect(canvas, o, d, cev, [&](const Hit& h) {
        if (nh == 0 || h.t < first.t) first = h;
        ++nh;
      });
    }
    if (nh > 0) {
      v.emit = true;
      v.x1 = (float)first.p.x;
      v.y1 = (float)first.p.y;
      v.hit = -1;
      v.flags = (uint8_t)((fl | (cev < INFINITY ? NEAR : 0u)) & 0xffu);
    }
  }
  // children: the next generation skips colours below the cutoff (tracer.rs:378-384)
  const bool deeper = (uint32_t)r.gen + 1 < sl.max_bounce;
  const float k0[4] = {__fmul_rn(r.c[0], v.f0), __fmul_rn(r.c[1], v.f0), __fmul_rn(r.c[2], v.f0), r.c[3]};
  const float k1[4] = {__fmul_rn(r.c[0], v.f1), __fmul_rn(r.c[1], v.f1), __fmul_rn(r.c[2], v.f1), r.c[3]};
  v.child0 = v.child0 && deeper && !below_cutoff(k0, sl.cutoff);
  v.child1 = v.child1 && deeper && !below_cutoff(k1, sl.cutoff);
}

// the segment of an emitting lane at its place in the ring
__device__ __forceinline__ void store_segment_x(const SceneDev& S, const TraceBufs& B, const BounceX& v, const RayRec& r,
                                                unsigned long long slot, uint32_t& my_near) {
  if (v.flags & LG_PATH_NEAR_DEGENERATE) ++my_near;
  if (slot >= B.seg_cap) return;
  float4* dst = reinterpret_cast<float4*>(B.segs + slot);
  dst[0] = make_float4(v.x0, v.y0, v.x1, v.y1);
  dst[1] = make_float4(r.c[0], r.c[1], r.c[2], r.c[3]);
  if (B.seg_scene) B.seg_scene[slot] = r.scene;
  if (S.record_paths) {
    lg_path_record pr;
    pr.path = r.path; pr.primary = r.prim; pr.light = r.light; pr.gen = r.gen;
    pr.flags = v.flags; pr.hit = v.hit; pr.source = LG_SRC_TRACE;
    B.paths[slot] = pr;
  }
}

// One generation of a small frame in one launch: a thread takes its ray through the search, the
// solve and the bounce.  A few thousand rays leave the GPU nearly empty whatever the order, and
// three launches with their lists and records cost more than the lost coherence: eight
// generations of a disc and a mirror (4096 primaries) take 127 us instead of 225, five of 12
// objects (12,000 primaries) 212 instead of 290.  Bound by the latency of the chain from a ray's
// record through its FP64 solve to its children, of which a warp has one and an SM few; 64
// threads a CTA spread the warps over all SMs.  The candidates are those of k_scan (the same
// tests in table order), so the hits are the same bits.
template <bool CULL>
__global__ void __launch_bounds__(SMALL_THREADS) k_small_x(SceneDev S, TraceBufs B, uint32_t gen, int smem_fits) {
  for (int k = 0; k < 3; ++k) stamp_start(B.ctr, gen, k);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  const uint64_t n_in = n_in_of(S, B, gen);
  if ((uint64_t)blockIdx.x * blockDim.x >= n_in) return;  // no ray for this CTA
  bool failed;
  const ObjScan* objs = stage_objects(S, reinterpret_cast<ObjScan*>(smem_raw), &bar, smem_fits != 0, B.ctr, failed);
  if (failed) return;
  const RayRec* qin = B.queue[gen & 1];
  RayRec* qout = B.queue[(gen + 1) & 1];
  const SceneLoc sl = scene_of<false>(S, 0u);
  uint32_t my_visits = 0, my_near = 0, my_tests = 0, my_cls = 0, my_solves = 0;
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  for (uint64_t base = warp * 32; base < n_in; base += nwarps * 32) {
    const uint64_t idx = base + lane_id();
    BounceX v;
    v.emit = v.child0 = v.child1 = false;
    v.flags = 0;
    v.hit = -1;
    v.f0 = v.f1 = 1.0f;
    RayRec r;
    bool live = idx < n_in;
    if (live) {
      if (gen == 0) primary_rec(S, idx, r);
      else r = qin[idx];
      live = !below_cutoff(r.c, sl.cutoff);
    }
    if (live) {
      ++my_visits;
      const V o = ray_o(r), d = ray_d(r);
      const float ox = (float)o.x, oy = (float)o.y, dx = (float)d.x, dy = (float)d.y;
      float thr = 3e38f, key[CAND], proved_t = INFINITY, proved_s = 0.0f;
      uint16_t cand[CAND];
      int nc = 0, leaf = -1, face = -1;
      ScanRec sc;
      sc.overflow = 0;
      for (uint32_t j = 0; j < S.n_obj; ++j) {
        float lb;
        ++my_tests;
        if (!bound_test(*reinterpret_cast<const float4*>(&objs[j]), ox, oy, dx, dy, thr, lb)) continue;
        ++my_cls;
        const Class32 c = classify32(objs[j], ox, oy, dx, dy, lb, j == r.src_obj ? (int)r.src_leaf : -1);
        if (c.ub < INFINITY) thr = fminf(thr, c.ub * (1.0f + 1e-4f) + 1e-4f);
        if (!(c.key <= thr)) continue;
        if (c.ub < proved_t) { proved_t = c.ub; leaf = c.leaf; face = c.face; proved_s = c.s; }
        if (nc == CAND) {  // full: drop candidates the bound has since excluded
          int w = 0;
          for (int k = 0; k < CAND; ++k)
            if (key[k] <= thr) { key[w] = key[k]; cand[w++] = cand[k]; }
          nc = w;
        }
        if (nc < CAND) { key[nc] = c.key; cand[nc++] = (uint16_t)j; }
        else sc.overflow = 1;
      }
      int m = 0;
      float k0 = INFINITY;
      for (int k = 0; k < nc; ++k)
        if (key[k] <= thr) {
          if (m == 0) k0 = key[k];
          cand[m++] = cand[k];
        }
      sc.nc = (uint8_t)m;
      HitRec hit;
      hit.obj = HIT_NONE;
      hit.flags = 0;
      if (m > 0 || sc.overflow) {
        bool done = false;
        if (m == 1 && !sc.overflow && leaf >= 0 && k0 == proved_t) {  // the only candidate's certain root
          const SolveRec& G = S.solve[cand[0]];
          lgx::Hit h;
          V n;
          if ((G.kind & 0xfu) != SR_TREE && solve_proved_x(G, o, d, leaf, face, proved_t, proved_s, h.t, h.p, n)) {
            store_hit_x(hit, (int)cand[0], h, n, leaf, INFINITY, 0);
            done = true;
            ++my_solves;
          }
        }
        if (!done) {
          Nearest N;
          const uint32_t count = sc.overflow ? S.n_obj : (uint32_t)m;
          for (uint32_t k = 0; k < count; ++k) {
            const uint32_t j = sc.overflow ? k : (uint32_t)cand[k];
            float lb;
            if (sc.overflow && !bound_test(*reinterpret_cast<const float4*>(&objs[j]), ox, oy, dx, dy, thr, lb)) continue;
            ++my_solves;
            N.consider(S, 0u, j, o, d);
          }
          N.store(S, 0u, d, sc.overflow ? LG_PATH_FALLBACK : 0, hit);
        }
      }
      bounce_x<false, CULL>(S, r, sc, &hit, v);
    }
    unsigned long long seg, s0, s1;
    reserve_out(B, gen, v.emit, v.child0, v.child1, seg, s0, s1);
    if (v.emit) store_segment_x(S, B, v, r, seg, my_near);
    if (v.child0 && s0 < B.queue_cap) store_child(qout + s0, r, child_x(r, v, v.d0, v.f0, r.path, r.medium));
    if (v.child1 && s1 < B.queue_cap)
      store_child(qout + s1, r, child_x(r, v, v.d1, v.f1, r.path | (1ull << r.gen), v.medium1));
  }
  stamp_end(B.ctr, gen);
  add_block_counts<5>({my_visits, my_near, my_tests, my_cls, my_solves},
                      {&B.ctr->visits, &B.ctr->near, &B.ctr->bound_tests, &B.ctr->object_tests, &B.ctr->fp64_solves});
}
template __global__ void k_small_x<false>(SceneDev, TraceBufs, uint32_t, int);
template __global__ void k_small_x<true>(SceneDev, TraceBufs, uint32_t, int);

template <bool MULTI, bool CULL>
__global__ void __launch_bounds__(256, LG_BOUNCE_X_BLOCKS) k_bounce_x(SceneDev S, TraceBufs B, uint32_t gen) {
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
  const RayRec* qin = B.queue[gen & 1];
  RayRec* qout = B.queue[(gen + 1) & 1];
  const unsigned lane = lane_id();
  const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = (gridDim.x * (uint64_t)blockDim.x) >> 5;
  uint32_t my_visits = 0, my_near = 0;
  for (uint64_t base = warp * 32; base < total; base += nwarps * 32) {
    const uint64_t i = base + lane;
    BounceX v;
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
      r = qin[idx];
      ++my_visits;
      bounce_x<MULTI, CULL>(S, r, sc, &B.hit[idx], v);
    }
    unsigned long long seg, s0, s1;
    reserve_out(B, gen, v.emit, v.child0, v.child1, seg, s0, s1);
    if (v.emit) store_segment_x(S, B, v, r, seg, my_near);
    if (v.child0 && s0 < B.queue_cap) store_child(qout + s0, r, child_x(r, v, v.d0, v.f0, r.path, r.medium));
    if (v.child1 && s1 < B.queue_cap)
      store_child(qout + s1, r, child_x(r, v, v.d1, v.f1, r.path | (1ull << r.gen), v.medium1));
  }
  stamp_end(B.ctr, gen);
  add_block_counts<2>({my_visits, my_near}, {&B.ctr->visits, &B.ctr->near});
}
template __global__ void k_bounce_x<false, false>(SceneDev, TraceBufs, uint32_t);
template __global__ void k_bounce_x<false, true>(SceneDev, TraceBufs, uint32_t);
template __global__ void k_bounce_x<true, false>(SceneDev, TraceBufs, uint32_t);
template __global__ void k_bounce_x<true, true>(SceneDev, TraceBufs, uint32_t);

}  // namespace lgd
