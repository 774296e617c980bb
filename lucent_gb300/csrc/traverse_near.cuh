// Nearest-first traversal with the reference's answers.
//
// The reference (intersectBVH, src/math/bvh.ts:265-320) visits left children
// first, whatever the ray's direction, so it tests many triangles that a
// nearest-first traversal never reaches, and reproducing its order means
// proving every one of its box tests. This file answers the same query in
// another order and proves the answer instead:
//
// What the reference returns. Let k be a triangle, t(k) its binary64
// Moller-Trumbore distance (ray.ts:22-45) and E(k), X(k) the binary64 entry
// (>= 0) and exit distances of its leaf's box (aabb.ts:84-98). In a tree whose
// boxes are nested, the reference tests k iff E(k) <= X(k) and E(k) <= c for
// the running closest distance c, and then takes it iff t(k) < c. Let w be the
// triangle of least t(k) over the leaves with E <= X, the lowest slot (first
// in the reference's order) among equals. If E(w) <= t(w), the reference
// returns w: until w is tested c > t(w) >= E(w), and nothing replaces w
// afterwards. If E(w) exceeds t(w) by rounding (flat boxes), the same holds as
// long as no other accepted triangle has its t in (t(w), E(w)].
//
// So the traversal may visit nodes in any order and skip any node that cannot
// hold a triangle with t <= t(w) (1 + 2^-16), the window that covers E(w); at
// the end it checks E(w) and, if two triangles met inside the window and E(w)
// is not clearly below them, hands the ray to the kernel that reproduces the
// reference's order (k_closest_wide_t, through a queue).
//
// When a node may be skipped. (1) Its box misses the ray. The reference's slab
// test of a leaf is evaluated in binary64; the binary32 test here uses, per
// axis, fma(b, inv, -(o inv)) with the products' rounding errors added to the
// entry and exit side (2^-22 |o inv| and 2^-20 relative), so whenever the
// reference's test of any leaf below passes, this one passes. (2) Its box
// begins beyond the window. That needs t(k) >= the entry distance of every box
// above k, which the reference's rounding does not guarantee: close to grazing
// incidence binary64's t, u, v are off, and the reference accepts points
// outside the triangle. The boxes of this view are therefore grown by what
// that error can be: the reference rejects |det| < 1e-12, and every numerator
// is off by at most 8 units (2^-53) of its absolute-value evaluation, so the
// accepted point o + t d lies within
//   1.03e-3 |e1| |e2| |d| (3 |s| + t |d| + |e1| + |e2|)
// of the triangle (1.03e-3 = 2^-50 x 1.155 / 1e-12; 1.155 bounds
// the norm of |a| x |b| by absolute values over |a| |b|; s = o - v0), which is
// microns for the triangles of a mesh. Triangles in an axis plane (walls,
// floors, most large ones) have det and t as single products of relative error
// 2^-48 |e1||e2| / |e1 x e2| and need almost none. leaf_growth() computes the
// bound for |d| <= 2 and origins within two diagonals of the tree's centre; for
// farther ones it rises linearly with the distance, and the ray's boxes are
// grown by the largest such rise of any triangle (NearTree::far), as long as
// that is small against a leaf. Other rays go to the ordered kernel, but for
// those that pass the root's boxes by. A tree
// with many leaves whose growth is not small against the scene (scenes in units
// far above 1, where 1e-12 is no bound at all), with boxes that are not nested
// or do not hold their triangles, nodes that the root never reaches or slots
// out of visiting order (caller-supplied trees), or with leaves of over 255
// triangles is not traversed this way (NearTree::usable).
//
// A record: (min.xyz, reference), (max.xyz, unused); the reference is the
// binary index of an inner node or kNearLeaf | first slot << 8 | count. As in
// the four-wide view, records 4 n .. 4 n + 3 are the grandchildren of binary
// node n, a leaf child standing in for its own (opening the child of largest
// surface twice instead measured the same within 1 %).
#pragma once
#include "traverse_wide.cuh"

namespace lucent {

constexpr int kNearLeaf = (int)0x80000000;
constexpr int kNearNone = kNearLeaf;  // a leaf of no triangles
constexpr int kNearMaxLeaf = 255;
constexpr float kNearWindow = 1.0000153f;      // 1 + 2^-16
constexpr float kNearSlack = 1.0000010f;       // 1 + 2^-20
constexpr float kNearOiPad = 2.3841858e-07f;   // 2^-22
// A warp tests boxes while a quarter of its lanes have some to test, then
// triangles (one a lane and turn) the same way, at most kNearSteps turns each;
// lanes whose ray is finished wait until a refill's worth of them write their
// answers and fetch rays together. Closest hit per 512 x 512 x 16 box frame and
// per 1080p x 4 frame over 2 M triangles: one box or leaf per lane and turn
// 3.27 and 13.4 ms; three boxes, then whole leaves, answers where they fall
// 2.70 and 10.4; in turns 2.40 and 9.4 (turns of 4 the same; ending below 12,
// 16 or 20 lanes up to 2 % slower; the loops unrolled 3.4 and 12.4, by their
// spills).
constexpr int kNearSteps = 8;
// Turns a warp takes at most between two refills; its rays are then handed to
// the ordered kernels (which count their own steps). A tree is walked once per
// ray, so this ends nothing sooner than a scene of many overlapping boxes.
constexpr uint32_t kNearTurns = 1u << 20;
// Any hit: one ray per thread without refill 2.35 ms of the box frame; in turns,
// with refills at 24 lanes: 1.57 at (128, 8), 7 blocks 1.62, 6 1.63; refill at
// 16 1.60.
constexpr int kAnyThreads = 128, kAnyBlocks = 8, kAnySteps = 8, kAnyRefill = 24;
// Norm-based bound of mt_classify's absolute-value evaluations: 2^-19 x 6 max|a| max|b| max|c|.
constexpr float kMtRel6 = 6.f * kMtRel;

// Triangle test against the window's end: kTriReject only if the reference
// certainly rejects or t is certainly at or beyond c; otherwise mt_classify's
// answer. Most triangles are rejected by a looser bound first, from the
// largest components of the factors (18 operations less per triangle than the
// absolute-value evaluations, which only the rest need).
LUCENT_DEV TriClass mt_classify_near(const Ray32& r, float md6, float4 a, float4 b, float4 c3, float tmin_lo,
                                     float tmin_hi, float c, float& t_lo, float& t_hi) {
  const float3 e1 = make_float3(b.x - a.x, b.y - a.y, b.z - a.z);
  const float3 e2 = make_float3(c3.x - a.x, c3.y - a.y, c3.z - a.z);
  const float3 d = r.d;
  const float3 p = make_float3(d.y * e2.z - d.z * e2.y, d.z * e2.x - d.x * e2.z, d.x * e2.y - d.y * e2.x);
  const float det = e1.x * p.x + e1.y * p.y + e1.z * p.z;
  const float3 s = make_float3(r.o.x - a.x, r.o.y - a.y, r.o.z - a.z);
  const float U = s.x * p.x + s.y * p.y + s.z * p.z;
  const float3 q = make_float3(s.y * e1.z - s.z * e1.y, s.z * e1.x - s.x * e1.z, s.x * e1.y - s.y * e1.x);
  const float V = d.x * q.x + d.y * q.y + d.z * q.z;
  const float m1 = fmaxf(fmaxf(fabsf(e1.x), fabsf(e1.y)), fabsf(e1.z));
  const float m2 = fmaxf(fmaxf(fabsf(e2.x), fabsf(e2.y)), fabsf(e2.z));
  const float ms = fmaxf(fmaxf(fabsf(s.x), fabsf(s.y)), fabsf(s.z));
  const float A = fabsf(det);
  const float sg = det < 0.f ? -1.f : 1.f;
  const float Ua = U * sg, Va = V * sg;
  {
    const float k2 = md6 * m2, k1 = md6 * m1;
    const float fD = fmaf(k2, m1, kAbsFloor), fU = fmaf(k2, ms, kAbsFloor), fV = fmaf(k1, ms, kAbsFloor);
    // With the sign of det unknown (A <= fD) nothing is decided here.
    if (A > fD && (Ua + fU < 0.f || Va + fV < 0.f || Ua + Va - (fU + fV) > A + fD)) return kTriReject;
  }
  const float T = e2.x * q.x + e2.y * q.y + e2.z * q.z;
  const float3 ad = make_float3(fabsf(d.x), fabsf(d.y), fabsf(d.z));
  const float3 ae1 = make_float3(fabsf(e1.x), fabsf(e1.y), fabsf(e1.z));
  const float3 ae2 = make_float3(fabsf(e2.x), fabsf(e2.y), fabsf(e2.z));
  const float3 as = make_float3(fabsf(s.x), fabsf(s.y), fabsf(s.z));
  const float3 ap = make_float3(ad.y * ae2.z + ad.z * ae2.y, ad.z * ae2.x + ad.x * ae2.z, ad.x * ae2.y + ad.y * ae2.x);
  const float3 aq = make_float3(as.y * ae1.z + as.z * ae1.y, as.z * ae1.x + as.x * ae1.z, as.x * ae1.y + as.y * ae1.x);
  const float eD = fmaf(ae1.x * ap.x + ae1.y * ap.y + ae1.z * ap.z, kMtRel, kAbsFloor);
  const float eU = fmaf(as.x * ap.x + as.y * ap.y + as.z * ap.z, kMtRel, kAbsFloor);
  const float eV = fmaf(ad.x * aq.x + ad.y * aq.y + ad.z * aq.z, kMtRel, kAbsFloor);
  const float eT = fmaf(ae2.x * aq.x + ae2.y * aq.y + ae2.z * aq.z, kMtRel, kAbsFloor);
  if (A + eD < 9.9e-13f) return kTriReject;  // |det| < 1e-12 for sure
  if (A <= eD) return kTriExact;
  const float Ta = T * sg;
  const float Ahi = __fadd_ru(A, eD), Alo = __fsub_rd(A, eD);
  if (Ua + eU < 0.f || Ua - eU > Ahi || Va + eV < 0.f || Ua + Va - (eU + eV) > Ahi) return kTriReject;
  if (Ta + eT < 0.f || Ta + eT <= tmin_lo * Alo * 0.99999905f) return kTriReject;  // t <= tMin
  if (Ta - eT >= c * Ahi * 1.00000095f) return kTriReject;                          // t >= c
  const bool inside = Ua - eU >= 0.f && Va - eV >= 0.f && Ua + Va + (eU + eV) <= Alo && Alo >= 1.0000001e-12f;
  if (!(inside && Ta - eT > tmin_hi * Ahi * 1.00000095f)) return kTriExact;
  t_lo = __fmul_rd(__fdiv_rd(__fsub_rd(Ta, eT), Ahi), 0.99999994f);
  t_hi = __fmul_ru(__fdiv_ru(__fadd_ru(Ta, eT), Alo), 1.00000012f);
  return kTriAccept;
}

// The ray as the box tests use it: per axis the reciprocal direction and
// o * inv moved outward by its rounding error for the entry and exit side.
struct NearRay {
  float3 inv, oe, ox;
};
// `grow`: how much the boxes are grown for this ray.
LUCENT_DEV NearRay make_near_ray(const Ray32& r, float grow) {
  NearRay n;
  n.inv = r.inv;
  const float3 oi = make_float3(r.o.x * r.inv.x, r.o.y * r.inv.y, r.o.z * r.inv.z);
  const float px = fmaf(fabsf(oi.x), kNearOiPad, grow * fabsf(r.inv.x));
  const float py = fmaf(fabsf(oi.y), kNearOiPad, grow * fabsf(r.inv.y));
  const float pz = fmaf(fabsf(oi.z), kNearOiPad, grow * fabsf(r.inv.z));
  n.oe = make_float3(oi.x + px, oi.y + py, oi.z + pz);
  n.ox = make_float3(oi.x - px, oi.y - py, oi.z - pz);
  return n;
}

// Entry distance (>= 0) of a record's box, and whether the ray may meet the
// box at a distance up to c (never false when the reference's binary64 test
// of a leaf inside would pass with closest distance c (1 - 2^-20) or less).
LUCENT_DEV bool near_box(const NearRay& n, float4 lo, float4 hi, float c, float& entry) {
  const bool bx = n.inv.x < 0.f, by = n.inv.y < 0.f, bz = n.inv.z < 0.f;
  const float ex = fmaf(bx ? hi.x : lo.x, n.inv.x, -n.oe.x), xx = fmaf(bx ? lo.x : hi.x, n.inv.x, -n.ox.x);
  const float ey = fmaf(by ? hi.y : lo.y, n.inv.y, -n.oe.y), xy = fmaf(by ? lo.y : hi.y, n.inv.y, -n.ox.y);
  const float ez = fmaf(bz ? hi.z : lo.z, n.inv.z, -n.oe.z), xz = fmaf(bz ? lo.z : hi.z, n.inv.z, -n.ox.z);
  entry = fmaxf(fmaxf(ex, ey), fmaxf(ez, 0.f));
  const float exit = fmaf(fminf(fminf(xx, xy), xz), kNearSlack, kAbsFloor);
  return entry <= fminf(exit, c);
}

// Two hits within the window of each other: the lesser binary64 t wins, the
// lower slot among equals. Returns the winner with exact bounds of its t.
struct NearBest {
  int slot;
  float lo, hi;
};
static __device__ __noinline__ NearBest near_tie(float3 o, float3 d, const float4* __restrict__ tris, double tmin,
                                                 int s0, int s1) {
  double t[2], u, v;
  for (int k = 0; k < 2; k++) {
    const float4* g = tris + 3 * (size_t)(k ? s1 : s0);
    t[k] = __longlong_as_double(0x7ff0000000000000ll);
    ts_triangle({o.x, o.y, o.z}, {d.x, d.y, d.z}, d3f(__ldg(g)), d3f(__ldg(g + 1)), d3f(__ldg(g + 2)), tmin,
                __longlong_as_double(0x7ff0000000000000ll), t[k], u, v);
  }
  const bool second = t[1] < t[0] || (t[1] == t[0] && s1 < s0);
  const double w = second ? t[1] : t[0];
  return {second ? s1 : s0, __double2float_rd(w), __double2float_ru(w)};
}

// A triangle test the binary32 bounds leave open, or one whose alpha needs the
// barycentrics: the reference's binary64 test in (tMin, tMax) and its alpha.
template <class Pol>
static __device__ __noinline__ bool near_exact(const Pol& P, int scene, uint32_t key, bool use_alpha, float3 o,
                                               float3 d, const float4* __restrict__ tris, int slot, double tmin,
                                               double tmax, float& lo, float& hi) {
  double t, u, v;
  const float4* g = tris + 3 * (size_t)slot;
  if (!ts_triangle({o.x, o.y, o.z}, {d.x, d.y, d.z}, d3f(__ldg(g)), d3f(__ldg(g + 1)), d3f(__ldg(g + 2)), tmin, tmax,
                   t, u, v))
    return false;
  if (use_alpha && !P.alpha(scene, slot, key, (float)u, (float)v)) return false;
  lo = __double2float_rd(t);
  hi = __double2float_ru(t);
  return true;
}

// Whether the reference's binary64 slab test of a leaf box passes at tMax.
static __device__ __noinline__ bool near_leaf_passes(float4 lo, float4 hi, float3 o, float3 d, double tMax) {
  return !ts_slab_culled(lo, hi, {o.x, o.y, o.z}, inv_exact(d), tMax);
}

// Whether the view covers the ray, and how much its boxes must be grown.
LUCENT_DEV bool near_ray_ok(float3 o, float3 d, const NearView& v, float& grow) {
  const float x = o.x - v.bound.x, y = o.y - v.bound.y, z = o.z - v.bound.z;
  const float dist = sqrtf(x * x + y * y + z * z);
  grow = fmaxf(dist - v.far.x, 0.f) * v.far.y;
  return safe_ray(o, d) && dist <= v.bound.w && d.x * d.x + d.y * d.y + d.z * d.z <= 4.f;
}

// Whether a ray that the view does not cover meets none of the root's boxes:
// with no box skipped for its distance, their test holds for every safe ray, as
// for any hit.
static __device__ __noinline__ bool near_misses_all(float3 o, float3 d, const Node* nodes, float c) {
  if (!safe_ray(o, d)) return false;
  const NearRay n = make_near_ray(make_ray32(o, d), 0.f);
  const float4* rec = reinterpret_cast<const float4*>(nodes);
  bool any = false;
#pragma unroll
  for (int i = 0; i < kWide; i++) {
    float e;
    any = near_box(n, __ldg(rec + 2 * i), __ldg(rec + 2 * i + 1), c, e) || any;
  }
  return !any;
}

// Closest hit: persistent warps, one ray per lane, refilled as in
// k_closest_wide_t. A turn tests four boxes (16 operations each instead
// of the 60 of a certain decision), sorts the hits by entry distance (the two
// low bits of the distance carry the record number) and goes on with the
// nearest. With few rays for the grid, a warp takes only as many as spread
// them over all warps: fewer lanes in a warp diverge less, and a launch of few
// rays lasts as long as its slowest warp.
// Bound by instruction issue on coherent waves (ncu, box frame, bounce 1: 18.0
// of 32 lanes active, issue slots 70 % busy, L1 64 %, DRAM 4 %), by L1 and
// divergence on incoherent rays (the soup: 13.0 lanes, L1 90 %, DRAM 0.4 %),
// by the longest ray's chain in small launches.
// Against the ordered wide kernel: 4,099 rays into 20,480 triangles 276 -> 69
// us a call, 10^6 rays into the 65,536-triangle soup 3.47 -> 1.80 ms, closest
// hit of the box frame (11.8 M rays, 82 k triangles) 4.19 -> 2.35 ms, of a
// 1080p 4-spp frame over 2 M triangles (14.7 M rays) 25.5 -> 9.0 ms.
template <class Pol>
__global__ void __launch_bounds__(Pol::kNearThreads, Pol::kNearBlocks) k_closest_near_t(TravArgs A, const __grid_constant__ Pol P) {
  wait_for_previous();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const float tmin_lo = __double2float_rd(A.tMin), tmin_hi = __double2float_ru(A.tMin);
  const float cmax_lo = __double2float_rd(A.tMax), cmax_hi = __double2float_ru(A.tMax);
  const uint32_t n = P.count();
  const bool use_alpha = P.alpha_any();
  const uint32_t warps = gridDim.x * (Pol::kNearThreads / 32);
  const int lanes = (int)min(32u, (n + warps - 1) / warps);
  const int refill = min(Pol::kNearRefill, lanes), turn = max(1, lanes / 4);

  bool has = false, exhausted = lane >= lanes;  // has: a ray whose answer is not written yet
  uint32_t ri = 0, key = 0;
  Ray32 r;
  NearRay nr;
  float md6 = 0.f, c = 0.f, lo = 0.f, hi = 0.f;
  int best = -1, pend = -1, sp = 0, ref = kNearNone;  // pend: a second hit inside the window, not yet compared
  NearView bv{};
  if constexpr (!Pol::kMultiScene) bv = A.near;
  WidePending stack[kWideStack];
  uint32_t turns = 0;

  auto pop = [&]() {
    while (sp > 0) {
      const WidePending e = stack[--sp];
      if (e.ehi <= c) return e.rec;
    }
    return kNearNone;
  };
  while (true) {
    const unsigned wait = __ballot_sync(FULL, ref == kNearNone && (has || !exhausted));
    const bool idle = __ballot_sync(FULL, ref != kNearNone) == 0;
    if (++turns > kNearTurns && ref != kNearNone) {
      A.queue[atomicAdd(A.queue_len, 1u)] = ri;
      has = false;
      ref = kNearNone;
    }
    if (__popc(wait) >= refill || idle) {
      turns = 0;
      // The answers of the lanes that wait, together.
      if (has && ref == kNearNone) {
        has = false;
        if (best < 0) {
          P.miss(ri);
        } else {
          const bool tie = pend >= 0;
          if (tie) {
            count_stat(A, 3);
            const NearBest b = near_tie(r.o, r.d, bv.tris, A.tMin, best, pend);
            best = b.slot;
            lo = b.lo;
          }
          const Node box = P.leaf_box(A, bv.scene, best);
          float ehi;
          const float INF32 = __int_as_float(0x7f800000);
          const SlabClass cl = classify_slab_e(r, box.lo, box.hi, INF32, INF32, ehi);
          bool ok = cl == kPass;
          if (cl == kAmbiguous) {
            count_stat(A, 1);
            ok = near_leaf_passes(box.lo, box.hi, r.o, r.d, __longlong_as_double(0x7ff0000000000000ll));
          }
          ok = ok && (ehi <= lo || (!tie && ehi * kNearSlack <= c && ehi <= cmax_lo));
          if (ok) P.finish(ri, best);
          else A.queue[atomicAdd(A.queue_len, 1u)] = ri;
        }
      }
      const bool need = ref == kNearNone && !exhausted;
      const unsigned m = __ballot_sync(FULL, need);
      if (m) {
        const int leader = __ffs(m) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(A.work, (uint32_t)__popc(m));
        base = __shfl_sync(FULL, base, leader);
        if (need) {
          ri = base + __popc(m & lt);
          if (ri >= n) {
            exhausted = true;
          } else {
            float3 o, d;
            P.ray(ri, o, d);
            if constexpr (Pol::kMultiScene) bv = P.near_view(ri);
            float grow;
            if (!near_ray_ok(o, d, bv, grow)) {
              // Rays past the tree end here: 10^6 of them from afar 94 us handed
              // on, 52 so (49 in the ordered kernels alone).
              if (near_misses_all(o, d, bv.nodes, cmax_hi * kNearSlack)) {
                count_stat(A, 0);
                P.miss(ri);
              } else {
                A.queue[atomicAdd(A.queue_len, 1u)] = ri;
              }
            } else {
              r = make_ray32(o, d);
              nr = make_near_ray(r, grow);
              md6 = kMtRel6 * fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
              key = use_alpha ? P.key(ri) : 0u;
              count_stat(A, 0);
              c = cmax_hi;
              best = -1;
              pend = -1;
              sp = 0;
              ref = 0;
              has = true;
            }
          }
        }
      }
      if (__ballot_sync(FULL, has) == 0 && __all_sync(FULL, exhausted)) break;
    }

    // Boxes.
#pragma unroll 1
    for (int it = 0; it < kNearSteps; it++) {
      if (ref >= 0) {
        if (sp + 3 > kWideStack) {  // unreachable for trees the reference's stack can traverse
          A.queue[atomicAdd(A.queue_len, 1u)] = ri;
          has = false;
          ref = kNearNone;
        } else {
          const float4* rec = reinterpret_cast<const float4*>(bv.nodes) + (size_t)ref * (2 * kWide);
          unsigned k[kWide];
          int rf[kWide];
#pragma unroll
          for (int i = 0; i < kWide; i++) {
            const float4 bl = __ldg(rec + 2 * i), bh = __ldg(rec + 2 * i + 1);
            float e;
            const bool hit = near_box(nr, bl, bh, c, e);
            k[i] = hit ? (__float_as_uint(e) & ~3u) | (unsigned)i : 0xffffffffu;
            rf[i] = __float_as_int(bl.w);
          }
          auto cas = [](unsigned& x, unsigned& y) {
            const unsigned a = min(x, y), b = max(x, y);
            x = a;
            y = b;
          };
          cas(k[0], k[1]);
          cas(k[2], k[3]);
          cas(k[0], k[2]);
          cas(k[1], k[3]);
          cas(k[1], k[2]);
          auto ref_of = [&](unsigned key4) {
            const int a = key4 & 1u ? rf[1] : rf[0], b = key4 & 1u ? rf[3] : rf[2];
            return key4 & 2u ? b : a;
          };
#pragma unroll
          for (int i = kWide - 1; i > 0; i--)
            if (k[i] != 0xffffffffu) stack[sp++] = {ref_of(k[i]), __uint_as_float(k[i] & ~3u)};
          ref = k[0] != 0xffffffffu ? ref_of(k[0]) : pop();
        }
      }
      if (__popc(__ballot_sync(FULL, ref >= 0)) < turn) break;
    }
    // Triangles, one a lane and turn: the reference counts down to the next.
#pragma unroll 1
    for (int it = 0; it < kNearSteps; it++) {
      if (ref < 0 && (ref & 255)) {
        const int slot = (ref & 0x7fffffff) >> 8;
        ref += 255;  // first + 1, count - 1
        const float4* g = bv.tris + 3 * (size_t)slot;
        float tl, th;
        const TriClass tc = mt_classify_near(r, md6, __ldg(g), __ldg(g + 1), __ldg(g + 2), tmin_lo, tmin_hi, c, tl, th);
        bool take = tc != kTriReject;
        if (take) {
          bool exact = tc == kTriExact || !(th < cmax_lo);
          if (use_alpha) {
            const AlphaAnswer aa = P.alpha_fast(bv.scene, slot, key);
            take = aa != kAlphaPass;
            exact = exact || aa == kAlphaDefer;  // a textured alpha needs the binary64 barycentrics
          }
          if (take && exact) {
            count_stat(A, 2);
            take = near_exact(P, bv.scene, key, use_alpha, r.o, r.d, bv.tris, slot, A.tMin, A.tMax, tl, th);
          }
        }
        if (take) {
          if (best < 0 || th * kNearWindow < lo) {
            best = slot;
            pend = -1;
            lo = tl;
            hi = th;
          } else if (!(tl > hi * kNearWindow)) {  // compared at the end, unless a nearer hit makes it moot
            if (pend >= 0) {
              count_stat(A, 3);
              const NearBest b = near_tie(r.o, r.d, bv.tris, A.tMin, best, pend);
              best = b.slot;
              lo = b.lo;
              hi = b.hi;
            }
            pend = slot;
            lo = fminf(lo, tl);
            hi = fminf(hi, th);
          }
          c = fminf(cmax_hi, hi * kNearWindow);
        }
        if (!(ref & 255)) ref = pop();
      }
      if (__popc(__ballot_sync(FULL, ref < 0 && (ref & 255))) < turn) break;
    }
  }
}

// Any hit: with the cull distance fixed at tMax the reference's answer is
// whether some triangle it accepts in (tMin, tMax) lies in a leaf whose
// binary64 slab test passes at tMax, in whatever order they are visited. The
// boxes are tested conservatively on the way down; the leaf's own test is made
// for an accepted triangle only.
template <class Pol>
__global__ void __launch_bounds__(kAnyThreads, kAnyBlocks) k_anyhit_near_t(TravArgs A, const __grid_constant__ Pol P) {
  wait_for_previous();
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const float tmin_lo = __double2float_rd(A.tMin), tmin_hi = __double2float_ru(A.tMin);
  const uint32_t n = P.count();
  const bool use_alpha = P.alpha_any();
  const uint32_t warps = gridDim.x * (kAnyThreads / 32);
  const int lanes = (int)min(32u, (n + warps - 1) / warps);
  const int refill = min(kAnyRefill, lanes), turn = max(1, lanes / 4);

  bool exhausted = lane >= lanes;
  uint32_t ri = 0, key = 0;
  Ray32 r;
  NearRay nr;
  float md6 = 0.f, tmax = 0.f;
  int sp = 0, ref = kNearNone;
  NearView bv = A.near;
  int stack[kWideStack];
  uint32_t turns = 0;
  while (true) {
    if (++turns > kNearTurns && ref != kNearNone) {
      A.queue[atomicAdd(A.queue_len, 1u)] = ri;
      ref = kNearNone;
    }
    const bool need = ref == kNearNone && !exhausted;
    const unsigned m = __ballot_sync(FULL, need);
    if (m && (__popc(m) >= refill || __ballot_sync(FULL, ref != kNearNone) == 0)) {
      turns = 0;
      const int leader = __ffs(m) - 1;
      uint32_t base = 0;
      if (lane == leader) base = atomicAdd(A.work, (uint32_t)__popc(m));
      base = __shfl_sync(FULL, base, leader);
      if (need) {
        ri = base + __popc(m & lt);
        if (ri >= n) {
          exhausted = true;
        } else {
          float3 o, d;
          P.ray(ri, o, d);
          if constexpr (Pol::kMultiScene) bv = P.near_view(ri);
          if (!safe_ray(o, d)) {
            A.queue[atomicAdd(A.queue_len, 1u)] = ri;
          } else {
            r = make_ray32(o, d);
            nr = make_near_ray(r, 0.f);  // nothing is skipped for its distance: no growth needed
            md6 = kMtRel6 * fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z));
            key = use_alpha ? P.key(ri) : 0u;
            tmax = P.tmax32(ri);
            sp = 0;
            ref = 0;
          }
        }
      }
    }
    if (__all_sync(FULL, exhausted && ref == kNearNone)) break;
#pragma unroll 1
    for (int it = 0; it < kAnySteps; it++) {
      if (ref >= 0) {
        if (sp + 3 > kWideStack) {  // unreachable, as above
          A.queue[atomicAdd(A.queue_len, 1u)] = ri;
          ref = kNearNone;
        } else {
          const float4* rec = reinterpret_cast<const float4*>(bv.nodes) + (size_t)ref * (2 * kWide);
          const float c = tmax * kNearSlack;
          ref = kNearNone;
#pragma unroll
          for (int i = 0; i < kWide; i++) {
            const float4 bl = __ldg(rec + 2 * i), bh = __ldg(rec + 2 * i + 1);
            float e;
            if (!near_box(nr, bl, bh, c, e)) continue;
            if (ref != kNearNone) stack[sp++] = ref;
            ref = __float_as_int(bl.w);
          }
          if (ref == kNearNone && sp > 0) ref = stack[--sp];
        }
      }
      if (__popc(__ballot_sync(FULL, ref >= 0)) < turn) break;
    }
#pragma unroll 1
    for (int it = 0; it < kAnySteps; it++) {
      if (ref < 0 && (ref & 255)) {
        const int slot = (ref & 0x7fffffff) >> 8;
        ref += 255;  // first + 1, count - 1
        const float4* g = bv.tris + 3 * (size_t)slot;
        float tl, th;
        const TriClass tc =
            mt_classify_near(r, md6, __ldg(g), __ldg(g + 1), __ldg(g + 2), tmin_lo, tmin_hi, tmax, tl, th);
        bool take = tc != kTriReject;
        if (take) {
          bool exact = tc == kTriExact || !(th < tmax);
          if (use_alpha) {
            const AlphaAnswer aa = P.alpha_fast(bv.scene, slot, key);
            take = aa != kAlphaPass;
            exact = exact || aa == kAlphaDefer;
          }
          if (take && exact)
            take = near_exact(P, bv.scene, key, use_alpha, r.o, r.d, bv.tris, slot, A.tMin, (double)tmax, tl, th);
          if (take) {
            const Node box = P.leaf_box(A, bv.scene, slot);
            const SlabClass cl = classify_slab(r, box.lo, box.hi, tmax, tmax);
            take = cl == kPass || (cl == kAmbiguous && near_leaf_passes(box.lo, box.hi, r.o, r.d, (double)tmax));
          }
        }
        if (take) {
          P.shadow(ri, true);  // unoccluded rays need no answer
          ref = kNearNone;
        } else if (!(ref & 255)) {
          ref = sp > 0 ? stack[--sp] : kNearNone;
        }
      }
      if (__popc(__ballot_sync(FULL, ref < 0 && (ref & 255))) < turn) break;
    }
  }
}

}  // namespace lucent
