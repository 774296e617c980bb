// GPU binned-SAH BVH builder whose output equals the reference's buildBVH
// (src/math/bvh.ts:52-252): same node array, same triIndices permutation.
//
// Why the result is the reference's:
//  * every per-node quantity the reference computes is either an exact
//    reduction (min/max of binary32 values, integer counts), which any order
//    reproduces, or a binary64 decision: the bin of a centroid, the cheapest
//    split, whether splitting pays. Those are made in binary32 where its error
//    bound decides them, else in binary64 in the reference's own operation
//    order (this file is compiled with -fmad=false);
//  * the SAH choice is the reference's first strict minimum (axis-major, bin
//    ascending): a parallel argmin with ties broken by candidate index;
//  * the in-place partition (bvh.ts:126-140) is sequential, but its final
//    permutation has a closed form computable from prefix counts (see
//    partition_dest below);
//  * nodes are built in any order under temporary ids and renumbered at the
//    end: the k-th inner node in left-first DFS preorder owns children
//    (2k+1, 2k+2) (bvh.ts:238-242).
//
// Nodes above kSub triangles are split level by level, a block per chunk of
// kChunk triangles and five launches a level that find their work (tasks,
// chunks) on the device; each subtree of at most kSub triangles is then
// finished by one block in shared memory, a warp per node. Small builds take
// smaller subtrees and one launch for all big levels (k_big_levels). The host
// waits once for the last big level (not in small builds), once for the node
// count and once at the end.
// Figures (positions on the device): see k_subtree and gpu_build_bvh.
#include <cooperative_groups.h>

#include <cfloat>

#include "common.cuh"
#include "internal.h"

namespace lucent {
namespace build {

constexpr int kMaxBins = 32;
constexpr int kChunk = 1024;  // triangles per block of a big level, 4 a thread
// Triangles of a subtree that one block finishes: 65 KB of shared memory at 12
// bins, three blocks an SM.
constexpr int kSub = 1024;
constexpr int kSubThreads = 512;  // at most: see k_subtree's launch
constexpr int kCluster = 8, kLevelThreads = 512;  // blocks of k_big_levels and their threads

struct Prims {
  const float4* lo;  // (min.xyz, centroid.x)
  const float4* hi;  // (max.xyz, centroid.y)
  const float* cz;   // centroid.z
};

__device__ __forceinline__ unsigned ord(float f) {
  const unsigned b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unord(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// boxArea (bvh.ts:35-40), binary64, reference operation order.
__device__ __forceinline__ double box_area(double x0, double y0, double z0, double x1, double y1, double z1) {
  const double dx = x1 - x0, dy = y1 - y0, dz = z1 - z0;
  return dx < 0 ? 0.0 : 2 * ((dx * dy + dy * dz) + dz * dx);
}
__device__ __forceinline__ float box_area32(const float* b) {
  const float dx = b[3] - b[0], dy = b[4] - b[1], dz = b[5] - b[2];
  return dx < 0 ? 0.f : 2 * ((dx * dy + dy * dz) + dz * dx);
}

// Per-node split setup (bvh.ts:163-174): centroid bounds, the axes that are
// binned, and the binary32 scale of each.
struct Split {
  float cmin[3], cmax[3], scale[3];
  int axes;  // bit a: axis a is binned
};

// Extents in binary64 as the reference compares them; the comparisons are made
// in binary32 unless two extents (or one and 1e-9) are within its rounding.
static __device__ __noinline__ int split_axes_f64(const float* c, bool all) {
  const double e0 = (double)c[3] - (double)c[0], e1 = (double)c[4] - (double)c[1], e2 = (double)c[5] - (double)c[2];
  const int longest = e0 >= e1 && e0 >= e2 ? 0 : e1 >= e2 ? 1 : 2;
  const double e[3] = {e0, e1, e2};
  int axes = 0;
  for (int a = 0; a < 3; a++)
    if (e[a] > 1e-9 && (all || a == longest)) axes |= 1 << a;
  return axes;
}
__device__ __forceinline__ Split make_split(const float* cbox, uint32_t count, int bins) {
  Split s;
  float e[3];
  bool sure = true;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    s.cmin[a] = cbox[a];
    s.cmax[a] = cbox[3 + a];
    e[a] = cbox[3 + a] - cbox[a];
    s.scale[a] = __fdiv_rn((float)bins, e[a]);
    sure = sure && fabsf(e[a] - 1e-9f) > 1e-14f;
  }
  const bool all = count >= 512;
  auto apart = [](float x, float y) { return fabsf(x - y) > 9.5e-7f * fmaxf(fabsf(x), fabsf(y)); };
  sure = sure && (all || (apart(e[0], e[1]) && apart(e[0], e[2]) && apart(e[1], e[2])));
  if (sure) {
    const int longest = e[0] >= e[1] && e[0] >= e[2] ? 0 : e[1] >= e[2] ? 1 : 2;
    s.axes = 0;
#pragma unroll
    for (int a = 0; a < 3; a++)
      if (e[a] > 1e-9f && (all || a == longest)) s.axes |= 1 << a;
  } else {
    s.axes = split_axes_f64(cbox, all);
  }
  return s;
}

// binOf (bvh.ts:122-123). The binary32 value differs from the binary64 one by
// at most 4 roundings, 2.5e-7 of at most 32 bins; only next to an inner bin
// boundary can that change the bin (below 0 and above bins - 1 it is clamped).
static __device__ __noinline__ int bin_of_f64(float c, float cmin, float cmax, int bins) {
  const double scale = (double)bins / ((double)cmax - (double)cmin);
  const double f = floor(((double)c - (double)cmin) * scale);
  const int b = (int)fmin((double)(bins - 1), f);
  return b < 0 ? 0 : b;  // no-op for finite inputs (f >= 0); keeps any input in bounds
}
__device__ __forceinline__ int bin_of(const Split& s, float c, int a, int bins) {
  const float f = (c - s.cmin[a]) * s.scale[a], k = rintf(f);
  if (!(fabsf(f - k) > 1.2e-5f) && !(k < 0.5f) && !(k > (float)bins - 0.5f)) return bin_of_f64(c, s.cmin[a], s.cmax[a], bins);
  if (!(s.scale[a] > 1e-25f)) return bin_of_f64(c, s.cmin[a], s.cmax[a], bins);
  return min(bins - 1, max(0, (int)f));
}

__device__ __forceinline__ float cen_of(float4 lo, float4 hi, float cz, int a) { return a == 0 ? lo.w : a == 1 ? hi.w : cz; }

// Bins of one node, 7 words each: count, min xyz, max xyz (order-preserving uints).
__device__ __forceinline__ unsigned bin_clear(int w) { return w == 0 ? 0u : w < 4 ? 0xffffffffu : 0u; }
// Neighbouring triangles of a mesh fall into the same few bins, and atomics of
// many lanes on one address run one by one: with Grouped, a warp whose lanes
// (`act`) hold at most kGroups bins reduces each group first. The bins of the
// top level of a 2,000,000-triangle knot take 45 us so, 116 without; a soup's
// gain nothing, and the small nodes of a subtree lose (0.86 against 0.73 ms
// for a whole build of 82,000 triangles with six groups).
constexpr int kGroups = 3;
template <bool Grouped>
__device__ __forceinline__ void bins_add(unsigned* b, const Split& s, float4 lo, float4 hi, float cz, int bins,
                                         unsigned act, int lane) {
  const unsigned o[6] = {ord(lo.x), ord(lo.y), ord(lo.z), ord(hi.x), ord(hi.y), ord(hi.z)};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    if (!(s.axes >> a & 1)) continue;
    const int bin = bin_of(s, cen_of(lo, hi, cz, a), a, bins);
    unsigned* k = b + 7 * (a * bins + bin);
    unsigned peers = 0;
    bool lead = false, grouped = false;
    if constexpr (Grouped) {
      peers = __match_any_sync(act, bin);
      lead = lane == __ffs(peers) - 1;
      grouped = __popc(__ballot_sync(act, lead)) <= kGroups;
    }
    if (grouped) {
      unsigned r[6];
#pragma unroll
      for (int q = 0; q < 6; q++) r[q] = q < 3 ? __reduce_min_sync(peers, o[q]) : __reduce_max_sync(peers, o[q]);
      if (lead) {
        atomicAdd(k, (unsigned)__popc(peers));
#pragma unroll
        for (int q = 0; q < 6; q++) {
          if (q < 3) atomicMin(k + 1 + q, r[q]);
          else atomicMax(k + 1 + q, r[q]);
        }
      }
    } else {
      atomicAdd(k, 1u);
#pragma unroll
      for (int q = 0; q < 3; q++) {
        atomicMin(k + 1 + q, o[q]);
        atomicMax(k + 4 + q, o[3 + q]);
      }
    }
  }
}

// SAH sweep (bvh.ts:191-223) by one warp: lane b evaluates the splits after bin
// b; candidate c = a * (bins - 1) + b splits axis a after bin b. The
// reference keeps the first strict minimum in (a, b) order and splits if that
// is below the leaf's cost. Costs in binary32 first (9 roundings of positive
// terms: 5.4e-7): if one candidate is below every other by 4e-6 and clearly
// below or above the leaf's cost, that decides; else binary64 does.
struct Choice {
  int axis, bin;  // -1: no candidate
  uint32_t left_count;
  bool pays;      // cost below the leaf's
};

// The two sides of candidate (a, lane), and whether it is one: lane b holds bin
// b of axis a (at most 32), and prefix and suffix scans over the lanes give
// every split's boxes and counts at once. A split after an empty bin is the
// split before it again, so it cannot be the first minimum.
struct Sides {
  float l[6], r[6];
  uint32_t ln, rn;
  bool valid;
};
__device__ __forceinline__ Sides split_sides(const unsigned* bin, int a, int bins, int lane) {
  unsigned l[7], r[7];
  const bool in = lane < bins;
#pragma unroll
  for (int q = 0; q < 7; q++) l[q] = r[q] = in ? bin[7 * (a * bins + lane) + q] : bin_clear(q);
  const bool empty = l[0] == 0;
  for (int o = 1; o < bins; o <<= 1) {
#pragma unroll
    for (int q = 0; q < 7; q++) {
      const unsigned u = __shfl_up_sync(0xffffffffu, l[q], o), d = __shfl_down_sync(0xffffffffu, r[q], o);
      const unsigned x = lane >= o ? u : bin_clear(q), y = lane + o < 32 ? d : bin_clear(q);
      l[q] = q == 0 ? l[q] + x : q < 4 ? min(l[q], x) : max(l[q], x);
      r[q] = q == 0 ? r[q] + y : q < 4 ? min(r[q], y) : max(r[q], y);
    }
  }
  Sides s;
  s.ln = l[0];
  s.rn = __shfl_down_sync(0xffffffffu, r[0], 1);
#pragma unroll
  for (int q = 0; q < 6; q++) {
    s.l[q] = unord(l[1 + q]);
    s.r[q] = unord(__shfl_down_sync(0xffffffffu, r[1 + q], 1));
  }
  s.valid = lane < bins - 1 && !empty && s.rn > 0;
  return s;
}

// The decision in binary64, the reference's operations and order.
static __device__ __noinline__ Choice warp_sah_f64(const unsigned* bin, int axes, int bins, int lane, uint32_t count,
                                                   const float* box) {
  double best = __longlong_as_double(0x7ff0000000000000ll);
  int bestc = 0x7fffffff;
  uint32_t bestn = 0;
  for (int a = 0; a < 3; a++) {
    if (!(axes >> a & 1)) continue;
    const Sides s = split_sides(bin, a, bins, lane);
    if (!s.valid) continue;
    const int c = a * (bins - 1) + lane;
    const double la = box_area(s.l[0], s.l[1], s.l[2], s.l[3], s.l[4], s.l[5]);
    const double ra = box_area(s.r[0], s.r[1], s.r[2], s.r[3], s.r[4], s.r[5]);
    const double cost = la * (double)s.ln + ra * (double)s.rn;
    if (cost < best) {  // candidates of one lane arrive in increasing c
      best = cost;
      bestc = c;
      bestn = s.ln;
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double oc = __shfl_xor_sync(0xffffffffu, best, off);
    const int oi = __shfl_xor_sync(0xffffffffu, bestc, off);
    const uint32_t on = __shfl_xor_sync(0xffffffffu, bestn, off);
    if (oc < best || (oc == best && oi < bestc)) {
      best = oc;
      bestc = oi;
      bestn = on;
    }
  }
  if (bestc == 0x7fffffff) return {-1, -1, 0, false};
  const double leaf = (double)count * box_area(box[0], box[1], box[2], box[3], box[4], box[5]);
  return {bestc / (bins - 1), bestc % (bins - 1), bestn, !(best >= leaf)};
}

// `bin`, `count` and `box` are the warp's; every lane returns the same.
__device__ __forceinline__ Choice warp_sah(const unsigned* bin, int axes, int bins, int lane, uint32_t count,
                                           const float* box) {
  const float INF32 = __int_as_float(0x7f800000);
  float best = INF32, second = INF32;  // this lane's least and next cost
  int bestc = -1;
  uint32_t bestn = 0;
  bool any = false;
  for (int a = 0; a < 3; a++) {
    if (!(axes >> a & 1)) continue;
    const Sides s = split_sides(bin, a, bins, lane);
    if (!s.valid) continue;
    const int c = a * (bins - 1) + lane;
    any = true;
    const float cost = box_area32(s.l) * (float)s.ln + box_area32(s.r) * (float)s.rn;
    if (cost < best) {
      second = best;
      best = cost;
      bestc = c;
      bestn = s.ln;
    } else {
      second = fminf(second, cost);
    }
  }
  if (!__any_sync(0xffffffffu, any)) return {-1, -1, 0, false};
  // Costs are >= 0, so ordered as integers (overflows fail the range check below).
  const float least = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(best)));
  const float near = least * 1.000004f;
  const unsigned at = __ballot_sync(0xffffffffu, best <= near);
  const bool close = __any_sync(0xffffffffu, second <= near) || (at & (at - 1u));
  const float leaf = (float)count * box_area32(box);
  const bool sure = least > 1e-25f && least < 1e30f && leaf < 1e30f && fabsf(least - leaf) > 4e-6f * leaf;
  if (close || !sure) return warp_sah_f64(bin, axes, bins, lane, count, box);
  const int src = __ffs(at) - 1;
  const int c = __shfl_sync(0xffffffffu, bestc, src);
  const uint32_t ln = __shfl_sync(0xffffffffu, bestn, src);
  return {c / (bins - 1), c % (bins - 1), ln, least < leaf};
}

// Destination of the element at relative position r after the reference's
// in-place partition (bvh.ts:126-140). n elements, L left-goers, m = number
// of right-goers in [0, L) = number of left-goers in [L, n).
//   front left-goer            stays
//   k-th front right-goer      -> n-1 (k = 0) or Q[k-1]-1
//   j-th back left-goer (from the end) -> P[j]
//   back right-goer with a back left-goer below it -> r-1
//   other back right-goers     -> r-1, except r = L -> Q[m-1]-1 (or n-1 if m = 0)
// with P[k] the k-th front right-goer's position (ascending) and Q[j] the
// j-th back left-goer's position counted from the end (Q[j] = Qasc[m-1-j]).
// Returns n (an impossible destination) if the counts are inconsistent; the
// caller then raises the error word instead of writing out of bounds.
template <class T>
__device__ __forceinline__ uint32_t partition_dest(uint32_t r, bool left, uint32_t L, uint32_t n, uint32_t m,
                                                   uint32_t rank_fr, uint32_t rank_bl_asc, uint32_t bl_before,
                                                   const T* P, const T* Qasc) {
  uint32_t d;
  if (r < L) {
    if (left) return r;
    if (rank_fr == 0) return n - 1;
    if (rank_fr > m) return n;
    d = (uint32_t)Qasc[m - rank_fr] - 1u;
  } else if (left) {
    if (rank_bl_asc >= m) return n;
    d = (uint32_t)P[m - 1 - rank_bl_asc];
  } else if (bl_before > 0 || r != L) {
    return r - 1;
  } else {
    d = m > 0 ? (uint32_t)Qasc[0] - 1u : n - 1;
  }
  return d < n ? d : n;
}

struct Task {
  uint32_t start, end;
  int32_t node;
  int32_t src;  // which order buffer holds its triangles (Ctx::tri)
};

// A big node while its level is worked on.
struct Big {
  Task t;
  Split split;
  uint32_t chunk0, chunks;  // its chunks of the level
  int axis, bin;            // axis < 0: not partitioned (leaf, or split in the middle)
  int leaf;
  uint32_t mid;             // absolute
  int kid[2];               // big index of the children in the next level, -1: not big
};

struct Chunk {
  uint32_t big, begin, end;  // element range
};

enum : int { kNRec = 0, kNSmall, kErrW, kNBig, kNChunk = kNBig + 2, kCtrBuild = kNChunk + 2 };

struct Ctx {
  Prims p;
  uint32_t* tri[3];   // triangle order: two buffers that levels alternate between, and the final one
  float4* recs;       // nodes by temporary id, 2 float4: (min, first slot or left child), (max, count; 0 inner)
  uint32_t* parent;   // by temporary id, + 1 (0: none)
  uint32_t* ctr;      // kNRec ...
  Task* small;        // subtrees
  Big* big[2];        // by level parity
  unsigned* box[2];   // 12 words per big node: box and centroid box (order-preserving uints)
  unsigned* bins;     // 3 * bins * 7 words per big node, clear between levels
  Chunk* chunk[2];
  unsigned* bits;     // kChunk / 32 words per chunk: the triangle goes left
  uint2* count;       // per chunk: front right-goers, back left-goers
  int32_t *P, *Q;     // positions of front right-goers and back left-goers
  uint32_t n, big_cap, chunk_cap, rec_cap;
  uint32_t sub;       // triangles of a subtree, at most kSub
  int max_leaf, nbins;
};

__device__ __forceinline__ void write_rec(const Ctx& cx, int32_t id, const float* box, uint32_t first, uint32_t count) {
  cx.recs[2 * (size_t)id] = make_float4(box[0], box[1], box[2], __int_as_float((int)first));
  cx.recs[2 * (size_t)id + 1] = make_float4(box[3], box[4], box[5], __int_as_float((int)count));
}

__device__ __forceinline__ void box_of(const unsigned* w, float* box) {
#pragma unroll
  for (int q = 0; q < 6; q++) box[q] = unord(w[q]);
}

// Appends big node `t` to level parity `p` with its chunks (one warp). Returns
// its index, or -1 with the error word set.
__device__ __forceinline__ int push_big(const Ctx& cx, int p, Task t, int lane) {
  const uint32_t chunks = (t.end - t.start + kChunk - 1) / kChunk;
  uint32_t i = 0, c0 = 0;
  if (lane == 0) {
    i = atomicAdd(cx.ctr + kNBig + p, 1u);
    c0 = atomicAdd(cx.ctr + kNChunk + p, chunks);
  }
  i = __shfl_sync(0xffffffffu, i, 0);
  c0 = __shfl_sync(0xffffffffu, c0, 0);
  if (i >= cx.big_cap || c0 + chunks > cx.chunk_cap) {  // impossible: the capacities hold every partition of n
    if (lane == 0) atomicOr(cx.ctr + kErrW, kErrQueue);
    return -1;
  }
  for (uint32_t c = lane; c < chunks; c += 32)
    cx.chunk[p][c0 + c] = {i, t.start + c * kChunk, min(t.end, t.start + (c + 1) * kChunk)};
  if (lane < 12) cx.box[p][12 * (size_t)i + lane] = lane % 6 < 3 ? 0xffffffffu : 0u;
  if (lane == 0) {
    Big& B = cx.big[p][i];
    B.t = t;
    B.chunk0 = c0;
    B.chunks = chunks;
  }
  return (int)i;
}

__global__ void k_clear_bins(unsigned* bins, size_t n) {
  wait_for_previous();
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
    bins[k] = bin_clear((int)(k % 7));
}

__global__ void k_init(Ctx cx) {
  const int lane = threadIdx.x;
  const Task root = {0, cx.n, 0, 0};
  if (lane == 0) {
    cx.ctr[kNRec] = 1;
    cx.parent[0] = 0;
    cx.ctr[kNSmall] = cx.n <= cx.sub;
    if (cx.n <= cx.sub) cx.small[0] = root;
  }
  if (cx.n > cx.sub) push_big(cx, 0, root, lane);
}

// Adds a warp's 12 extrema (ordered uints; 3 minima and 3 maxima, twice) to 12 words.
__device__ __forceinline__ void add_box(unsigned* to, const unsigned* v, int lane) {
#pragma unroll
  for (int q = 0; q < 12; q++) {
    const unsigned r = q % 6 < 3 ? __reduce_min_sync(0xffffffffu, v[q]) : __reduce_max_sync(0xffffffffu, v[q]);
    if (lane == 0) {
      if (q % 6 < 3) atomicMin(to + q, r);
      else atomicMax(to + q, r);
    }
  }
}
__device__ __forceinline__ void clear_box(unsigned* v) {
#pragma unroll
  for (int q = 0; q < 12; q++) v[q] = q % 6 < 3 ? 0xffffffffu : 0u;
}
__device__ __forceinline__ void grow_box(unsigned* v, float4 lo, float4 hi, float cz) {
  const float x[6] = {lo.x, lo.y, lo.z, hi.x, hi.y, hi.z}, c[3] = {lo.w, hi.w, cz};
#pragma unroll
  for (int q = 0; q < 3; q++) {
    v[q] = min(v[q], ord(x[q]));
    v[3 + q] = max(v[3 + q], ord(x[3 + q]));
    const unsigned o = ord(c[q]);
    v[6 + q] = min(v[6 + q], o);
    v[9 + q] = max(v[9 + q], o);
  }
}

// ---------------------------------------------------------------------------
// Per-triangle bounds and centroids (bvh.ts:59-73), the identity order and the
// root's boxes.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_prim_bounds(const float* __restrict__ pos, Ctx cx, float4* __restrict__ lo4,
                                                     float4* __restrict__ hi4, float* __restrict__ cz) {
  wait_for_previous();
  __shared__ unsigned sbox[12];
  if (threadIdx.x < 12) sbox[threadIdx.x] = threadIdx.x % 6 < 3 ? 0xffffffffu : 0u;
  __syncthreads();
  unsigned v[12];
  clear_box(v);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cx.n; i += gridDim.x * blockDim.x) {
    const float* p = pos + (size_t)i * 9;
    float lo[3], hi[3], c[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float p0 = p[a], p1 = p[3 + a], p2 = p[6 + a];
      lo[a] = fminf(p0, fminf(p1, p2));
      hi[a] = fmaxf(p0, fmaxf(p1, p2));
      c[a] = __double2float_rn(((double)lo[a] + (double)hi[a]) * 0.5);
    }
    const float4 l4 = make_float4(lo[0], lo[1], lo[2], c[0]), h4 = make_float4(hi[0], hi[1], hi[2], c[1]);
    lo4[i] = l4;
    hi4[i] = h4;
    cz[i] = c[2];
    cx.tri[0][i] = i;
    grow_box(v, l4, h4, c[2]);
  }
  if (cx.n <= cx.sub) return;
  add_box(sbox, v, threadIdx.x & 31);
  __syncthreads();
  if (threadIdx.x < 12) {
    unsigned* to = cx.box[0] + threadIdx.x;
    if (threadIdx.x % 6 < 3) atomicMin(to, sbox[threadIdx.x]);
    else atomicMax(to, sbox[threadIdx.x]);
  }
}

// ---------------------------------------------------------------------------
// One level of big nodes (parity p): bins per chunk, decision per node, then
// the partition of the nodes that split at a bin: which side each triangle
// goes to, the lists of those that change halves, and the move into the other
// order buffer, which also gathers the children's boxes. Grids cover the most
// chunks and nodes a level can have; blocks beyond the level's own end at once.
// ---------------------------------------------------------------------------
template <int T>
__device__ __forceinline__ void big_bins(const Ctx& cx, int p, uint32_t chunk, unsigned* sbin) {
  const Chunk ck = cx.chunk[p][chunk];
  const unsigned* bx = cx.box[p] + 12 * (size_t)ck.big;
  float cbox[6];
  box_of(bx + 6, cbox);
  const Task t = cx.big[p][ck.big].t;
  const Split s = make_split(cbox, t.end - t.start, cx.nbins);
  const int words = 3 * cx.nbins * 7;
  for (int k = threadIdx.x; k < words; k += T) sbin[k] = bin_clear(k % 7);
  __syncthreads();
  const uint32_t* tri = cx.tri[t.src];
#pragma unroll
  for (int j = 0; j < kChunk / T; j++) {
    const uint32_t i = ck.begin + j * T + threadIdx.x;
    const unsigned act = __ballot_sync(0xffffffffu, i < ck.end);
    if (i < ck.end) {
      const uint32_t k = tri[i];
      bins_add<true>(sbin, s, __ldg(cx.p.lo + k), __ldg(cx.p.hi + k), __ldg(cx.p.cz + k), cx.nbins, act, threadIdx.x & 31);
    }
  }
  __syncthreads();
  unsigned* to = cx.bins + (size_t)ck.big * words;
  for (int k = threadIdx.x; k < words; k += T) {
    const int w = k % 7;
    if (sbin[k - w] == 0) continue;  // an empty bin
    if (w == 0) atomicAdd(to + k, sbin[k]);
    else if (w < 4) atomicMin(to + k, sbin[k]);
    else atomicMax(to + k, sbin[k]);
  }
}

__global__ void __launch_bounds__(256) k_big_bins(Ctx cx, int p) {
  wait_for_previous();
  extern __shared__ unsigned sbin[];
  if (blockIdx.x == 0 && threadIdx.x == 0) cx.ctr[kNBig + (p ^ 1)] = cx.ctr[kNChunk + (p ^ 1)] = 0;
  if (blockIdx.x < cx.ctr[kNChunk + p]) big_bins<256>(cx, p, blockIdx.x, sbin);
}

// One warp per big node w: split, children, the node's record; its bins are left clear.
__device__ __forceinline__ void big_sah(const Ctx& cx, int p, uint32_t w, unsigned* bin, int lane) {
  Big& B = cx.big[p][w];
  const Task t = B.t;
  const uint32_t count = t.end - t.start;
  const int words = 3 * cx.nbins * 7;
  for (int k = lane; k < words; k += 32) {
    unsigned* from = cx.bins + (size_t)w * words + k;
    bin[k] = *from;
    *from = bin_clear(k % 7);
  }
  __syncwarp();
  float box[6], cbox[6];
  box_of(cx.box[p] + 12 * (size_t)w, box);
  box_of(cx.box[p] + 12 * (size_t)w + 6, cbox);
  const Split s = make_split(cbox, count, cx.nbins);
  Choice ch{-1, -1, 0, false};
  bool leaf = count <= (uint32_t)cx.max_leaf;  // bvh.ts:157-160
  if (!leaf) {
    ch = warp_sah(bin, s.axes, cx.nbins, lane, count, box);
    if (!ch.pays && count <= (uint32_t)cx.max_leaf * 4) leaf = true;  // bvh.ts:227-232
  }
  uint32_t mid = ch.pays ? t.start + ch.left_count : (t.start + t.end) >> 1;
  if (mid == t.start || mid == t.end) mid = (t.start + t.end) >> 1;  // bvh.ts:236
  uint32_t id = 0;
  if (!leaf) {
    if (lane == 0) id = atomicAdd(cx.ctr + kNRec, 2u);
    id = __shfl_sync(0xffffffffu, id, 0);
    if (id + 2 > cx.rec_cap) {  // impossible for non-empty children; never write past recs
      if (lane == 0) atomicOr(cx.ctr + kErrW, kErrQueue);
      leaf = true;
    }
  }
  if (lane == 0) {
    write_rec(cx, t.node, box, leaf ? t.start : id, leaf ? count : 0u);
    B.split = s;
    B.axis = leaf || !ch.pays ? -1 : ch.axis;
    B.bin = ch.bin;
    B.leaf = leaf;
    B.mid = mid;
  }
  for (int k = 0; k < 2; k++) {
    int kid = -1;
    if (!leaf) {
      const Task c = {k ? mid : t.start, k ? t.end : mid, (int32_t)id + k, t.src ^ 1};
      if (lane == 0) cx.parent[id + k] = (uint32_t)t.node + 1;
      if (c.end - c.start > cx.sub) kid = push_big(cx, p ^ 1, c, lane);
      else if (lane == 0) cx.small[atomicAdd(cx.ctr + kNSmall, 1u)] = c;  // at most n tasks: children are not empty
    }
    if (lane == 0) B.kid[k] = kid;
  }
}

__global__ void __launch_bounds__(128) k_big_sah(Ctx cx, int p) {
  wait_for_previous();
  extern __shared__ unsigned sbin[];
  const int warp = threadIdx.x >> 5;
  const uint32_t w = blockIdx.x * 4 + warp;
  if (w < cx.ctr[kNBig + p]) big_sah(cx, p, w, sbin + warp * 3 * cx.nbins * 7, threadIdx.x & 31);
}

// Which side each triangle of a chunk goes to (bits), and how many cross.
template <int T>
__device__ __forceinline__ void big_count(const Ctx& cx, int p, uint32_t chunk) {
  __shared__ uint32_t cross[2];
  const Chunk ck = cx.chunk[p][chunk];
  const Big& B = cx.big[p][ck.big];
  if (B.axis < 0) return;
  if (threadIdx.x < 2) cross[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint32_t* tri = cx.tri[B.t.src];
#pragma unroll
  for (int j = 0; j < kChunk / T; j++) {
    const uint32_t i = ck.begin + j * T + threadIdx.x;
    bool left = false;
    if (i < ck.end) {
      const uint32_t k = tri[i];
      const float c = B.axis == 0 ? __ldg(&cx.p.lo[k].w) : B.axis == 1 ? __ldg(&cx.p.hi[k].w) : __ldg(cx.p.cz + k);
      left = bin_of(B.split, c, B.axis, cx.nbins) <= B.bin;
    }
    const unsigned m = __ballot_sync(0xffffffffu, left);
    const unsigned fr = __ballot_sync(0xffffffffu, i < ck.end && i < B.mid && !left);
    const unsigned bl = __ballot_sync(0xffffffffu, i < ck.end && i >= B.mid && left);
    if (lane == 0) {
      cx.bits[(size_t)chunk * (kChunk / 32) + j * (T / 32) + (threadIdx.x >> 5)] = m;
      if (fr) atomicAdd(&cross[0], __popc(fr));
      if (bl) atomicAdd(&cross[1], __popc(bl));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) cx.count[chunk] = make_uint2(cross[0], cross[1]);
}
__global__ void __launch_bounds__(256) k_big_count(Ctx cx, int p) {
  wait_for_previous();
  if (blockIdx.x < cx.ctr[kNChunk + p]) big_count<256>(cx, p, blockIdx.x);
}

// Block-wide setup of a partitioned chunk: the crossing counts before it and
// over the whole node, and before each of its 32 words. All threads call it.
struct Cross {
  uint32_t fr0, bl0, m, m2;
};
template <int T>
__device__ __forceinline__ Cross cross_setup(const Ctx& cx, const Big& B, const Chunk& ck, uint32_t chunk, unsigned* word,
                                             uint2* before) {
  __shared__ uint32_t sum[4];
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 4) sum[threadIdx.x] = 0;
  __syncthreads();
  uint32_t v[4] = {0, 0, 0, 0};  // before this chunk, and in all
  for (uint32_t c = threadIdx.x; c < B.chunks; c += T) {
    const uint2 k = cx.count[B.chunk0 + c];
    v[2] += k.x;
    v[3] += k.y;
    if (B.chunk0 + c < chunk) {
      v[0] += k.x;
      v[1] += k.y;
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t s = __reduce_add_sync(0xffffffffu, v[q]);
    if (lane == 0 && s) atomicAdd(&sum[q], s);
  }
  if (threadIdx.x < kChunk / 32) {  // one warp: word `lane` covers elements begin + 32 lane ...
    const unsigned m = cx.bits[(size_t)chunk * (kChunk / 32) + lane];
    const uint32_t b = ck.begin + 32 * lane;
    const uint32_t len = b < ck.end ? min(32u, ck.end - b) : 0u, front = b < B.mid ? min(len, B.mid - b) : 0u;
    auto low = [](uint32_t k) { return k >= 32 ? 0xffffffffu : (1u << k) - 1u; };
    const uint32_t fr = __popc(~m & low(front)), bl = __popc(m & low(len) & ~low(front));
    uint32_t a = fr, c = bl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, a, o), y = __shfl_up_sync(0xffffffffu, c, o);
      if (lane >= o) {
        a += x;
        c += y;
      }
    }
    word[lane] = m;
    before[lane] = make_uint2(a - fr, c - bl);
  }
  __syncthreads();
  return {sum[0], sum[1], sum[2], sum[3]};
}
// Ranks of element i among the node's front right-goers and back left-goers.
struct Rank {
  bool left, front;
  uint32_t fr, bl;
};
__device__ __forceinline__ Rank rank_of(const Cross& X, const Big& B, const Chunk& ck, uint32_t i, const unsigned* word,
                                        const uint2* before) {
  const uint32_t r = i - ck.begin, j = r >> 5, l = r & 31;
  const unsigned m = word[j], lt = (1u << l) - 1u;
  const uint32_t b = ck.begin + 32 * j, front = b < B.mid ? min(32u, B.mid - b) : 0u;
  const unsigned in_front = front >= 32 ? 0xffffffffu : (1u << front) - 1u;
  return {(m >> l & 1u) != 0, i < B.mid, X.fr0 + before[j].x + __popc(~m & in_front & lt),
          X.bl0 + before[j].y + __popc(m & ~in_front & lt)};
}

template <int T>
__device__ __forceinline__ void big_place(const Ctx& cx, int p, uint32_t chunk) {
  __shared__ unsigned word[kChunk / 32];
  __shared__ uint2 before[kChunk / 32];
  const Chunk ck = cx.chunk[p][chunk];
  const Big& B = cx.big[p][ck.big];
  if (B.axis < 0) return;
  const Cross X = cross_setup<T>(cx, B, ck, chunk, word, before);
  if (X.m != X.m2 && threadIdx.x == 0) atomicOr(cx.ctr + kErrW, kErrQueue);  // impossible for a consistent binning
#pragma unroll
  for (int j = 0; j < kChunk / T; j++) {
    const uint32_t i = ck.begin + j * T + threadIdx.x;
    if (i >= ck.end) continue;
    const Rank k = rank_of(X, B, ck, i, word, before);
    const uint32_t r = i - B.t.start;
    if (k.front && !k.left) cx.P[B.t.start + k.fr] = (int32_t)r;
    if (!k.front && k.left) cx.Q[B.t.start + k.bl] = (int32_t)r;
  }
}

__global__ void __launch_bounds__(256) k_big_place(Ctx cx, int p) {
  wait_for_previous();
  if (blockIdx.x < cx.ctr[kNChunk + p]) big_place<256>(cx, p, blockIdx.x);
}

template <int T>
__device__ __forceinline__ void big_move(const Ctx& cx, int p, uint32_t chunk) {
  __shared__ unsigned word[kChunk / 32], sbox[2][12];
  __shared__ uint2 before[kChunk / 32];
  const Chunk ck = cx.chunk[p][chunk];
  const Big& B = cx.big[p][ck.big];
  const uint32_t* tri = cx.tri[B.t.src];
  uint32_t* to = cx.tri[B.leaf ? 2 : B.t.src ^ 1];
  const bool kids = B.kid[0] >= 0 || B.kid[1] >= 0;
  if (threadIdx.x < 24) sbox[threadIdx.x / 12][threadIdx.x % 12] = threadIdx.x % 6 < 3 ? 0xffffffffu : 0u;
  Cross X{0, 0, 0, 0};
  if (B.axis >= 0) X = cross_setup<T>(cx, B, ck, chunk, word, before);
  else __syncthreads();
  const uint32_t start = B.t.start, n = B.t.end - start, L = B.mid - start;
  unsigned v[2][12];
  clear_box(v[0]);
  clear_box(v[1]);
#pragma unroll
  for (int j = 0; j < kChunk / T; j++) {
    const uint32_t i = ck.begin + j * T + threadIdx.x;
    if (i >= ck.end) continue;
    const uint32_t t = tri[i], r = i - start;
    bool left = r < L;
    uint32_t d = r;
    if (B.axis >= 0) {
      const Rank k = rank_of(X, B, ck, i, word, before);
      left = k.left;
      d = partition_dest(r, k.left, L, n, X.m, k.fr, k.bl, k.bl, cx.P + start, cx.Q + start);
      if (d >= n) {
        atomicOr(cx.ctr + kErrW, kErrQueue);
        d = r;
      }
    }
    to[start + d] = t;
    if (kids) {
      const float4 lo = __ldg(cx.p.lo + t), hi = __ldg(cx.p.hi + t);
      const float cz = __ldg(cx.p.cz + t);
      if (left) grow_box(v[0], lo, hi, cz);
      else grow_box(v[1], lo, hi, cz);
    }
  }
  if (!kids) return;
  for (int k = 0; k < 2; k++)
    if (B.kid[k] >= 0) add_box(sbox[k], v[k], threadIdx.x & 31);
  __syncthreads();
  if (threadIdx.x < 24) {
    const int k = threadIdx.x / 12, q = threadIdx.x % 12;
    if (B.kid[k] >= 0) {
      unsigned* b = cx.box[p ^ 1] + 12 * (size_t)B.kid[k] + q;
      if (q % 6 < 3) atomicMin(b, sbox[k][q]);
      else atomicMax(b, sbox[k][q]);
    }
  }
}
__global__ void __launch_bounds__(256) k_big_move(Ctx cx, int p) {
  wait_for_previous();
  if (blockIdx.x < cx.ctr[kNChunk + p]) big_move<256>(cx, p, blockIdx.x);
}

// All levels of a small build's big nodes by one cluster: the five steps of a
// level wait for one another at the cluster's barrier instead of at launches,
// and there are as many levels as the tree has, so subtrees can be small and
// many. Bound by its dependent loads (25 us a level of 2,503 triangles, where
// five launches took 30 to 45 and the empty levels 13 each). 512 threads a
// block against 256: whole builds of 12,000 triangles of a soup and a knot 519
// -> 490 and 571 -> 525 us, of 2,503 alike. A block a node, whose steps wait for the block alone, once
// nodes have a chunk each: within 3 % either way.
__global__ void __launch_bounds__(kLevelThreads) __cluster_dims__(kCluster, 1, 1) k_big_levels(Ctx cx) {
  wait_for_previous();
  extern __shared__ unsigned sbin[];
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const uint32_t rank = cluster.block_rank(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile const uint32_t* ctr = cx.ctr;
  // Every level makes its nodes smaller, so there are fewer than n; as many at
  // most as the launches' loop allows.
  for (int level = 0, p = 0;; level++, p ^= 1) {
    const uint32_t nodes = ctr[kNBig + p], chunks = ctr[kNChunk + p];
    if (nodes == 0) return;
    if (level == 8192) {
      if (rank == 0 && threadIdx.x == 0) atomicOr(cx.ctr + kErrW, kErrQueue);
      return;
    }
    if (rank == 0 && threadIdx.x == 0) cx.ctr[kNBig + (p ^ 1)] = cx.ctr[kNChunk + (p ^ 1)] = 0;
    for (uint32_t c = rank; c < chunks; c += kCluster) {
      big_bins<kLevelThreads>(cx, p, c, sbin);
      __syncthreads();
    }
    cluster.sync();
    for (uint32_t w = rank * (kLevelThreads / 32) + warp; w < nodes; w += kCluster * (kLevelThreads / 32)) {
      big_sah(cx, p, w, sbin + warp * 3 * cx.nbins * 7, lane);
      __syncwarp();
    }
    cluster.sync();
    for (uint32_t c = rank; c < chunks; c += kCluster) {
      big_count<kLevelThreads>(cx, p, c);
      __syncthreads();
    }
    cluster.sync();
    for (uint32_t c = rank; c < chunks; c += kCluster) {
      big_place<kLevelThreads>(cx, p, c);
      __syncthreads();
    }
    cluster.sync();
    for (uint32_t c = rank; c < chunks; c += kCluster) {
      big_move<kLevelThreads>(cx, p, c);
      __syncthreads();
    }
    cluster.sync();
  }
}

// ---------------------------------------------------------------------------
// One subtree per block, in shared memory: its triangles' bounds, their order
// and the nodes of the current level, a warp per node. Bound by the warps'
// dependent chains of shared-memory passes over nodes of a few triangles
// (before: a launch per level, a warp per node, every pass gathering from
// L2 and a binary64 division and sweep per node).
// ---------------------------------------------------------------------------
struct SubNode {
  uint16_t start, count;
  int32_t id;
};
inline size_t sub_bytes(uint32_t sub, int bins, int threads) {
  return (size_t)sub * (16 + 16 + 4 + 4 + 4 * 2) + (size_t)sub * sizeof(SubNode) + (size_t)threads / 32 * 3 * bins * 7 * 4;
}

struct Sub {
  float4 *lo, *hi;
  float* cz;
  uint32_t* gid;
  uint16_t *ord, *tmp, *P, *Q;
  SubNode* level[2];  // sub / 2 each: a node of the lists has two triangles or more
  unsigned* bins;     // this warp's
};

__device__ __forceinline__ void sub_box(const Sub& S, uint32_t start, uint32_t count, int lane, float* box) {
  unsigned v[6];
#pragma unroll
  for (int q = 0; q < 6; q++) v[q] = q < 3 ? 0xffffffffu : 0u;
  for (uint32_t i = lane; i < count; i += 32) {
    const uint32_t t = S.ord[start + i];
    const float4 lo = S.lo[t], hi = S.hi[t];
    v[0] = min(v[0], ord(lo.x)), v[1] = min(v[1], ord(lo.y)), v[2] = min(v[2], ord(lo.z));
    v[3] = max(v[3], ord(hi.x)), v[4] = max(v[4], ord(hi.y)), v[5] = max(v[5], ord(hi.z));
  }
#pragma unroll
  for (int q = 0; q < 6; q++)
    box[q] = unord(q < 3 ? __reduce_min_sync(0xffffffffu, v[q]) : __reduce_max_sync(0xffffffffu, v[q]));
}

// Splits one node with a warp (bvh.ts:150-242); children of more than
// max_leaf triangles go to `next`, the others are written as leaves.
__device__ __forceinline__ void sub_node(const Ctx& cx, const Sub& S, const Task& task, SubNode nd, int lane,
                                         uint32_t* next_id, uint32_t id_end, SubNode* next, uint32_t* n_next) {
  const uint32_t start = nd.start, count = nd.count;
  unsigned v[12];
  clear_box(v);
  for (uint32_t i = lane; i < count; i += 32) {
    const uint32_t t = S.ord[start + i];
    grow_box(v, S.lo[t], S.hi[t], S.cz[t]);
  }
  float box[6], cbox[6];
#pragma unroll
  for (int q = 0; q < 12; q++) {
    const float f = unord(q % 6 < 3 ? __reduce_min_sync(0xffffffffu, v[q]) : __reduce_max_sync(0xffffffffu, v[q]));
    if (q < 6) box[q] = f;
    else cbox[q - 6] = f;
  }
  const Split s = make_split(cbox, count, cx.nbins);
  const int per = cx.nbins * 7;
#pragma unroll
  for (int a = 0; a < 3; a++)
    if (s.axes >> a & 1)
      for (int k = lane; k < per; k += 32) S.bins[a * per + k] = bin_clear(k % 7);
  __syncwarp();
  if (s.axes)
    for (uint32_t i = lane; i < count; i += 32) {
      const uint32_t t = S.ord[start + i];
      bins_add<false>(S.bins, s, S.lo[t], S.hi[t], S.cz[t], cx.nbins, 0, lane);
    }
  __syncwarp();
  const Choice ch = warp_sah(S.bins, s.axes, cx.nbins, lane, count, box);
  __syncwarp();
  uint32_t id = 0;
  bool leaf = !ch.pays && count <= (uint32_t)cx.max_leaf * 4;  // bvh.ts:227-232
  if (!leaf) {
    if (lane == 0) id = atomicAdd(next_id, 2u);
    id = __shfl_sync(0xffffffffu, id, 0);
    if (id + 2 > id_end) {  // impossible for non-empty children; never write past recs
      if (lane == 0) atomicOr(cx.ctr + kErrW, kErrQueue);
      leaf = true;
    }
  }
  if (lane == 0) write_rec(cx, nd.id, box, leaf ? task.start + start : id, leaf ? count : 0u);
  if (leaf) return;
  uint32_t L = ch.pays ? ch.left_count : 0;
  if (ch.pays) {
    // Partition (bvh.ts:126-140): positions of the triangles that change
    // halves, then every triangle's destination.
    const unsigned lt = (1u << lane) - 1u;
    uint16_t *P = S.P + start, *Q = S.Q + start;
    auto goes_left = [&](uint32_t t) {
      return bin_of(s, cen_of(S.lo[t], S.hi[t], S.cz[t], ch.axis), ch.axis, cx.nbins) <= ch.bin;
    };
    uint32_t m = 0, bl = 0;
    for (uint32_t base = 0; base < count; base += 32) {
      const uint32_t r = base + lane;
      const bool left = r < count && goes_left(S.ord[start + r]);
      const bool is_fr = r < count && r < L && !left, is_bl = r >= L && left;
      const unsigned mf = __ballot_sync(0xffffffffu, is_fr), mb = __ballot_sync(0xffffffffu, is_bl);
      if (is_fr) P[m + __popc(mf & lt)] = (uint16_t)r;
      if (is_bl) Q[bl + __popc(mb & lt)] = (uint16_t)r;
      m += __popc(mf);
      bl += __popc(mb);
    }
    if (m != bl && lane == 0) atomicOr(cx.ctr + kErrW, kErrQueue);  // impossible for a consistent binning
    __syncwarp();
    uint32_t fr = 0;
    bl = 0;
    for (uint32_t base = 0; base < count; base += 32) {
      const uint32_t r = base + lane;
      const uint32_t t = r < count ? S.ord[start + r] : 0u;
      const bool left = r < count && goes_left(t);
      const bool is_fr = r < count && r < L && !left, is_bl = r >= L && left;
      const unsigned mf = __ballot_sync(0xffffffffu, is_fr), mb = __ballot_sync(0xffffffffu, is_bl);
      if (r < count) {
        const uint32_t rfr = fr + __popc(mf & lt), rbl = bl + __popc(mb & lt);
        uint32_t d = partition_dest(r, left, L, count, m, rfr, rbl, rbl, P, Q);
        if (d >= count) {
          atomicOr(cx.ctr + kErrW, kErrQueue);
          d = r;
        }
        S.tmp[start + d] = (uint16_t)t;
      }
      fr += __popc(mf);
      bl += __popc(mb);
    }
    __syncwarp();
    for (uint32_t r = lane; r < count; r += 32) S.ord[start + r] = S.tmp[start + r];
    __syncwarp();
  }
  const uint32_t a0 = task.start + start;
  uint32_t mid = ch.pays ? L : ((a0 + a0 + count) >> 1) - a0;  // the middle of absolute positions, as the reference takes it
  if (mid == 0 || mid == count) mid = ((a0 + a0 + count) >> 1) - a0;  // bvh.ts:236
  for (int k = 0; k < 2; k++) {
    const uint32_t cs = k ? start + mid : start, cc = k ? count - mid : mid;
    if (lane == 0) cx.parent[id + k] = (uint32_t)nd.id + 1;
    if (cc <= (uint32_t)cx.max_leaf) {  // bvh.ts:157-160
      float cb[6];
      sub_box(S, cs, cc, lane, cb);
      if (lane == 0) write_rec(cx, (int32_t)id + k, cb, task.start + cs, cc);
    } else if (lane == 0) {
      next[atomicAdd(n_next, 1u)] = {(uint16_t)cs, (uint16_t)cc, (int32_t)id + k};
    }
  }
}

__device__ __forceinline__ void subtree(const Ctx& cx, const Sub& S, const Task task, int warp, int lane) {
  __shared__ uint32_t n_level[2], next_id, id_end;
  const uint32_t n = task.end - task.start;
  const uint32_t* src = cx.tri[task.src] + task.start;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    const uint32_t t = src[i];
    S.gid[i] = t;
    S.lo[i] = __ldg(cx.p.lo + t);
    S.hi[i] = __ldg(cx.p.hi + t);
    S.cz[i] = __ldg(cx.p.cz + t);
    S.ord[i] = (uint16_t)i;
  }
  const bool one = n <= (uint32_t)cx.max_leaf;
  if (threadIdx.x == 0) {
    n_level[0] = !one;
    n_level[1] = 0;
    S.level[0][0] = {0, (uint16_t)n, task.node};
    // The subtree has at most 2 n - 1 nodes, its root's id is given; unused ids stay holes.
    const uint32_t want = one ? 0u : 2 * n - 2;
    next_id = want ? atomicAdd(cx.ctr + kNRec, want) : 0u;
    id_end = min(next_id + want, cx.rec_cap);
  }
  __syncthreads();
  if (one && warp == 0) {
    float box[6];
    sub_box(S, 0, n, lane, box);
    if (lane == 0) write_rec(cx, task.node, box, task.start, n);
  }
  for (int cur = 0; n_level[cur] > 0; cur ^= 1) {  // at most n levels: every node is split into smaller ones
    const uint32_t m = n_level[cur];
    for (uint32_t w = warp; w < m; w += blockDim.x / 32)
      sub_node(cx, S, task, S.level[cur][w], lane, &next_id, id_end, S.level[cur ^ 1], &n_level[cur ^ 1]);
    __syncthreads();
    if (threadIdx.x == 0) n_level[cur] = 0;
    __syncthreads();
  }
  uint32_t* to = cx.tri[2] + task.start;
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) to[i] = S.gid[S.ord[i]];
}

__global__ void __launch_bounds__(kSubThreads) k_subtree(Ctx cx) {
  wait_for_previous();
  const uint32_t tasks = cx.ctr[kNSmall];  // may be more than the grid has blocks

  extern __shared__ float4 smem[];
  Sub S;
  S.lo = smem;
  S.hi = S.lo + cx.sub;
  S.cz = (float*)(S.hi + cx.sub);
  S.gid = (uint32_t*)(S.cz + cx.sub);
  S.ord = (uint16_t*)(S.gid + cx.sub);
  S.tmp = S.ord + cx.sub;
  S.P = S.tmp + cx.sub;
  S.Q = S.P + cx.sub;
  S.level[0] = (SubNode*)(S.Q + cx.sub);
  S.level[1] = S.level[0] + cx.sub / 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  S.bins = (unsigned*)(S.level[1] + cx.sub / 2) + warp * 3 * cx.nbins * 7;
  for (uint32_t k = blockIdx.x; k < tasks; k += gridDim.x) {
    subtree(cx, S, cx.small[k], warp, lane);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Renumbering (bvh.ts:238-242): inner-node counts and heights bottom-up, then
// each inner node's DFS preorder rank (left = parent + 1, right = parent + 1 +
// inner nodes of the left subtree) by walking up, and its children's records
// at 2 rank + 1 and 2 rank + 2. Ids never used are holes (count -1).
// The way up is a chain of loads and one atomic a level: with what the next
// level needs loaded before the atomic, and the atomic ordering the counts by
// itself instead of two fences, 17 us for 2,503 triangles where it took 27.
// ---------------------------------------------------------------------------
__global__ void k_tree_counts(Ctx cx, uint32_t* __restrict__ arrived, uint32_t* inner, uint32_t* height,
                              uint32_t n_ids) {
  wait_for_previous();
  uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n_ids || __float_as_int(cx.recs[2 * (size_t)x + 1].w) <= 0) return;  // holes and inner nodes
  for (uint32_t up = cx.parent[x]; up != 0;) {  // the second child to arrive at a node goes on; ids fall on the way up
    x = up - 1;
    const uint32_t l = (uint32_t)__float_as_int(cx.recs[2 * (size_t)x].w);
    up = cx.parent[x];
    if (arrive(arrived + x) == 0) return;
    const uint32_t n = __ldcg(inner + l) + __ldcg(inner + l + 1), h = max(__ldcg(height + l), __ldcg(height + l + 1));
    __stcg(inner + x, 1 + n);
    __stcg(height + x, 1 + h);
  }
}

// `nodes`: device layout; `ref`: the reference's 8 floats (either may be null).
__global__ void k_tree_emit(Ctx cx, const uint32_t* __restrict__ inner, uint32_t n_ids, float4* __restrict__ nodes,
                            float4* __restrict__ ref) {
  const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= n_ids) return;
  const int cnt = __float_as_int(cx.recs[2 * (size_t)x + 1].w);
  auto emit = [&](uint32_t at, uint32_t id, uint32_t rank) {
    float4 lo = cx.recs[2 * (size_t)id], hi = cx.recs[2 * (size_t)id + 1];
    const int count = __float_as_int(hi.w), first = count > 0 ? __float_as_int(lo.w) : (int)(2 * rank + 1);
    if (nodes) {
      lo.w = __int_as_float(first);
      nodes[2 * (size_t)at] = lo;
      nodes[2 * (size_t)at + 1] = hi;
    }
    if (ref) {
      lo.w = (float)first;
      hi.w = (float)count;
      ref[2 * (size_t)at] = lo;
      ref[2 * (size_t)at + 1] = hi;
    }
  };
  if (x == 0) emit(0, 0, 0);
  if (cnt != 0) return;  // leaves and holes own no children
  uint32_t rank = 0;
  for (uint32_t y = x, up = cx.parent[y]; up != 0; y = up - 1, up = cx.parent[y]) {
    const uint32_t l = (uint32_t)__float_as_int(cx.recs[2 * (size_t)(up - 1)].w);
    rank += y == l ? 1u : 1u + inner[l];
  }
  const uint32_t l = (uint32_t)__float_as_int(cx.recs[2 * (size_t)x].w);
  emit(2 * rank + 1, l, rank + 1);
  emit(2 * rank + 2, l + 1, rank + 1 + inner[l]);
}

}  // namespace build
}  // namespace lucent

#include "bvh_build_host.inl"
