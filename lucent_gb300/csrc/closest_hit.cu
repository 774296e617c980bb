// BVH API instantiation of the shared traversal kernels (traverse.cuh):
// rays as 6 floats (or doubles) each, results per ray, hit ids equal to the
// reference's intersectBVH (src/math/bvh.ts:265-320).
#include "internal.h"
#include "traverse_near.cuh"

namespace lucent {

__device__ __forceinline__ void load_ray6(const float* rays, uint32_t i, float3& o, float3& d) {
  const float2* r2 = reinterpret_cast<const float2*>(rays) + (size_t)i * 3;
  const float2 a = __ldg(r2), b = __ldg(r2 + 1), c = __ldg(r2 + 2);
  o = make_float3(a.x, a.y, b.x);
  d = make_float3(b.y, c.x, c.y);
}

// Rays from a float array; results in prim/t/u/v (binary64 values rounded to
// binary32). The triangle's source index sits in v0.w.
struct ApiPolicy {
  const float* rays;
  uint32_t n;
  const float4* tris;
  int32_t* prim;
  float *tout, *uout, *vout;
  double tmin;
  __device__ uint32_t count() const { return n; }
  __device__ void ray(uint32_t k, float3& o, float3& d) const { load_ray6(rays, k, o, d); }
  __device__ uint32_t key(uint32_t) const { return 0; }
  static constexpr bool kMultiScene = false;
  static constexpr int kThreads = 128, kMinBlocks = 7;  // closest-hit block shape
  // Lanes of a wide-kernel warp that wait before it fetches new rays
  // (measured on 10^6 random rays into a 65,536-triangle soup: 4 over 1, 8, 16).
  static constexpr int kRefillMin = 4;
    // (7 blocks, 72 registers: the soup's 10^6 rays 1.82 ms, 1.90 at 8 blocks)
  static constexpr int kNearThreads = 128, kNearBlocks = 7, kNearRefill = 4;
  __device__ Node leaf_box(const TravArgs& A, int, int slot) const { return load_node(A.nodes, __ldg(A.leaf_of + slot)); }
  __device__ bool alpha(int, int, uint32_t, float, float) const { return true; }
  __device__ AlphaAnswer alpha_fast(int, int, uint32_t) const { return kAlphaBlock; }
  __device__ bool alpha_any() const { return false; }
  // The hit triangle, encoded -3 - slot until k_refine_api computes its
  // values with the warp converged (lanes finish their rays at different
  // steps, so per-ray arithmetic here would run one lane at a time).
  __device__ void finish(uint32_t k, int slot) const { prim[k] = -3 - slot; }
  __device__ void hit(uint32_t k, int slot, double t, double u, double v) const {
    prim[k] = __float_as_int(__ldg(tris + 3 * (size_t)slot).w);
    if (tout) tout[k] = __double2float_rn(t);
    if (uout) uout[k] = __double2float_rn(u);
    if (vout) vout[k] = __double2float_rn(v);
  }
  __device__ void miss(uint32_t k) const {
    prim[k] = -1;
    if (tout) tout[k] = __int_as_float(0x7f800000);
    if (uout) uout[k] = 0.f;
    if (vout) vout[k] = 0.f;
  }
  __device__ void fail(uint32_t k) const { prim[k] = -2; }
};

// f64-ray API: rays as 6 doubles, outputs in binary64 (always the exact path).
__global__ void k_closest_exact_d(TravArgs A, const double* __restrict__ rays, uint32_t n, int32_t* __restrict__ prim,
                                  double* __restrict__ tout, double* __restrict__ uout, double* __restrict__ vout) {
  ApiPolicy P{};
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double* r = rays + (size_t)i * 6;
    int slot;
    double t = 0, u = 0, v = 0;
    if (!trace_exact(A, P, bvh_of(A, P, i), {r[0], r[1], r[2]}, {r[3], r[4], r[5]}, 0, slot, t, u, v)) {
      prim[i] = -2;
    } else if (slot < 0) {
      prim[i] = -1;
      tout[i] = __longlong_as_double(0x7ff0000000000000ll);
      uout[i] = vout[i] = 0;
    } else {
      prim[i] = __float_as_int(__ldg(A.tris + 3 * (size_t)slot).w);
      tout[i] = t;
      uout[i] = u;
      vout[i] = v;
    }
  }
}

// A few binary64 rays (picks), a warp each. One thread's walk is a chain of
// dependent loads and binary64 tests, one pick into 81,920 triangles 200 to 650
// us a call, 1,000 rays 1.9 to 3.0 ms (here: 100 us, and 0.17 to 0.2 ms, of which
// the tree's depth in dependent steps is the most). The warp pops up to 32 pending nodes at a time and tests their
// children, or a leaf's triangles, a lane each. Nothing is skipped for its
// distance, so every triangle the reference could take is met; the answer is
// the one of least t (lowest slot among equals) if the reference reaches it:
// it visits a leaf iff every box on the way passes with the running closest
// c, and c > t(w) until w is tested, so it takes w if the largest entry
// distance on the way is at most t(w), or at least below the next t (the
// argument of traverse_near.cuh, here over any tree, as each box is tested).
// Rays with a zero or non-finite component (whose NaN slab decisions are not
// monotone), pending nodes beyond the list, equal least t or an undecided
// winner take one lane's walk in the reference's order instead.
constexpr int kPickPending = 768;
struct PickArgs {  // rays as kernel arguments: no copy to the device
  double r[kPickArgs * 6];
  __device__ const double* at(uint32_t k) const { return r + 6 * k; }
};
struct PickArray {
  const double* r;
  __device__ const double* at(uint32_t k) const { return r + 6 * (size_t)k; }
};
struct PendingBox {
  double entry;  // largest entry distance on the way
  int node;
  int pad;
};

// AABB.intersect's test (ts_slab_culled) with the entry distance it computes.
__device__ __forceinline__ bool slab_entry(const Node& nd, const double o[3], const double inv[3], double tMax,
                                           double& entry) {
  const double lo[3] = {(double)nd.lo.x, (double)nd.lo.y, (double)nd.lo.z};
  const double hi[3] = {(double)nd.hi.x, (double)nd.hi.y, (double)nd.hi.z};
  double tmin = 0, tmax = tMax;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double a = dmul(dsub(lo[i], o[i]), inv[i]), b = dmul(dsub(hi[i], o[i]), inv[i]);
    const double t0 = a > b ? b : a, t1 = a > b ? a : b;
    if (t0 > tmin) tmin = t0;
    if (t1 < tmax) tmax = t1;
  }
  entry = tmin;
  return !(tmax < tmin);
}

template <class Rays>
__global__ void __launch_bounds__(32) k_pick(TravArgs A, const __grid_constant__ Rays rays, PickHit* __restrict__ out) {
  __shared__ PendingBox list[kPickPending];
  const int lane = threadIdx.x;
  const uint32_t k = blockIdx.x;
  const double* r = rays.at(k);
  const double o[3] = {r[0], r[1], r[2]}, d[3] = {r[3], r[4], r[5]};
  const double inv[3] = {ddiv(1.0, d[0]), ddiv(1.0, d[1]), ddiv(1.0, d[2])};
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 3; i++) ok = ok && isfinite(o[i]) && isfinite(d[i]) && isfinite(inv[i]) && inv[i] != 0.0;
  const double INF64 = __longlong_as_double(0x7ff0000000000000ll);
  double bt = INF64, bu = 0, bv = 0, be = 0, second = INF64;  // this lane's least t, its entry distance, its next t
  int bs = 0x7fffffff;
  uint32_t n = 0, seen = 0;
  if (ok) {
    const Node root = load_node(A.nodes, 0);
    double e;
    if (slab_entry(root, o, inv, A.tMax, e)) {
      if (lane == 0) list[0] = {e, 0, 0};
      n = 1;
    }
  }
  __syncwarp();
  while (ok && n > 0) {
    const uint32_t take = min(n, 32u);
    seen += take;
    const bool mine = lane < (int)take;
    PendingBox it{};
    if (mine) it = list[n - 1 - lane];
    n -= take;
    __syncwarp();
    double e0 = 0, e1 = 0;
    bool p0 = false, p1 = false;
    int first = 0;
    if (mine) {
      const Node nd = load_node(A.nodes, it.node);
      const int cnt = node_count(nd);
      first = node_first(nd);
      if (cnt == 0) {
        const Node c0 = load_node(A.nodes, first), c1 = load_node(A.nodes, first + 1);
        p0 = slab_entry(c0, o, inv, A.tMax, e0);
        p1 = slab_entry(c1, o, inv, A.tMax, e1);
      }
      for (int q = 0; q < cnt; q++) {
        const int s = first + q;
        double t, u, v;
        if (!ts_triangle({o[0], o[1], o[2]}, {d[0], d[1], d[2]}, d3f(__ldg(A.tris + 3 * (size_t)s)),
                         d3f(__ldg(A.tris + 3 * (size_t)s + 1)), d3f(__ldg(A.tris + 3 * (size_t)s + 2)), A.tMin,
                         A.tMax, t, u, v))
          continue;
        if (t < bt || (t == bt && s < bs)) {
          second = bt;
          bt = t, bu = u, bv = v, bs = s, be = it.entry;
        } else if (t < second) {
          second = t;
        }
      }
    }
    const unsigned m0 = __ballot_sync(0xffffffffu, p0), m1 = __ballot_sync(0xffffffffu, p1);
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t push = __popc(m0) + __popc(m1);
    ok = n + push <= kPickPending && seen <= A.node_limit;  // (a tree is walked once)
    if (ok) {
      if (p0) list[n + __popc(m0 & lt)] = {fmax(it.entry, e0), first, 0};
      if (p1) list[n + __popc(m0) + __popc(m1 & lt)] = {fmax(it.entry, e1), first + 1, 0};
    }
    n += push;
    __syncwarp();
  }
  // The warp's least (t, slot), then the least t of all the others.
  double wt = bt;
  int ws = bs;
  for (int off = 16; off > 0; off >>= 1) {
    const double t = __shfl_xor_sync(0xffffffffu, wt, off);
    const int s = __shfl_xor_sync(0xffffffffu, ws, off);
    if (t < wt || (t == wt && s < ws)) wt = t, ws = s;
  }
  double next = bs == ws ? second : bt;
  for (int off = 16; off > 0; off >>= 1) next = fmin(next, __shfl_xor_sync(0xffffffffu, next, off));
  const bool hit = ws != 0x7fffffff, winner = hit && bs == ws;
  const double entry = __shfl_sync(0xffffffffu, be, hit ? __ffs(__ballot_sync(0xffffffffu, winner)) - 1 : 0);
  ok = ok && (!hit || (wt < next && (entry <= wt || entry < next)));
  PickHit h{INF64, 0, 0, -1, 0u};
  if (ok) {
    if (hit ? !winner : lane != 0) return;
    if (hit) h = {bt, bu, bv, __float_as_int(__ldg(A.tris + 3 * (size_t)bs).w), 0u};
  } else {
    if (lane != 0) return;
    __shared__ unsigned err;
    err = 0;
    int slot;
    TravArgs B = A;
    B.err = &err;
    ApiPolicy P{};
    if (!trace_exact(B, P, bvh_of(B, P, k), {o[0], o[1], o[2]}, {d[0], d[1], d[2]}, 0, slot, h.t, h.u, h.v)) {
      h.prim = -2;
    } else if (slot >= 0) {
      h.prim = __float_as_int(__ldg(A.tris + 3 * (size_t)slot).w);
    } else {
      h.t = INF64;
      h.u = h.v = 0;
    }
    h.err = err;
  }
  out[k] = h;
}

// The values of the hits the traversal found (prim = -3 - slot): the
// reference's binary64 t, u, v rounded to binary32, from double-float
// arithmetic where its bound proves the roundings of all three, else from
// binary64; prim becomes the triangle's source index. One thread per ray.
__global__ void k_refine_api(ApiPolicy P) {
  wait_for_previous();
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < P.n; k += gridDim.x * blockDim.x) {
    const int32_t code = P.prim[k];
    if (code > -3) continue;
    const int slot = -3 - code;
    float3 o, d;
    P.ray(k, o, d);
    const float4 a = __ldg(P.tris + 3 * (size_t)slot), b = __ldg(P.tris + 3 * (size_t)slot + 1),
                 c = __ldg(P.tris + 3 * (size_t)slot + 2);
    float3 tuv;
    if (tri_df32(o, d, a, b, c, true, tuv)) {
      P.hit(k, slot, tuv.x, tuv.y, tuv.z);
    } else {
      const Tri64 h = tri_f64(o, d, a, b, c, P.tmin, __longlong_as_double(0x7ff0000000000000ll));
      P.hit(k, slot, h.t, h.u, h.v);
    }
  }
}

// Reference nodes (8 floats, leftFirst/count as floats) -> device Node layout.
__global__ void k_pack_nodes(const float* __restrict__ ref, uint32_t count, Node* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const float* r = ref + (size_t)i * 8;
    Node nd;
    nd.lo = make_float4(r[0], r[1], r[2], __int_as_float((int)r[3]));
    nd.hi = make_float4(r[4], r[5], r[6], __int_as_float((int)r[7]));
    out[i] = nd;
  }
}

// Triangles gathered into leaf (slot) order, source index in v0.w.
__global__ void k_gather_tris(const float* __restrict__ pos, const uint32_t* __restrict__ tri_indices,
                              uint32_t tri_count, float4* __restrict__ out) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < tri_count; s += gridDim.x * blockDim.x) {
    const uint32_t src = tri_indices[s];
    const float* p = pos + (size_t)src * 9;
    out[3 * (size_t)s] = make_float4(p[0], p[1], p[2], __int_as_float((int)src));
    out[3 * (size_t)s + 1] = make_float4(p[3], p[4], p[5], 0.f);
    out[3 * (size_t)s + 2] = make_float4(p[6], p[7], p[8], 0.f);
  }
}

// Inverse of the two kernels above: back to the reference's layout.
__global__ void k_unpack(const Node* __restrict__ nodes, uint32_t count, const float4* __restrict__ tris,
                         uint32_t tri_count, float* __restrict__ ref, uint32_t* __restrict__ tri_indices) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count || i < tri_count; i += gridDim.x * blockDim.x) {
    if (i < count) {
      const Node nd = nodes[i];
      float* r = ref + (size_t)i * 8;
      r[0] = nd.lo.x, r[1] = nd.lo.y, r[2] = nd.lo.z, r[3] = (float)node_first(nd);
      r[4] = nd.hi.x, r[5] = nd.hi.y, r[6] = nd.hi.z, r[7] = (float)node_count(nd);
    }
    if (i < tri_count) tri_indices[i] = (uint32_t)__float_as_int(tris[3 * (size_t)i].w);
  }
}

int grid_for(uint32_t n, int block) {
  int g = (int)((n + block - 1) / block);
  return g < 1 ? 1 : (g > 65535 * 16 ? 65535 * 16 : g);
}

int persistent_blocks(const void* kernel, int block) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, block, 0);
  return (sms > 0 ? sms : 152) * (per > 0 ? per : 2);
}

void launch_pack_nodes(const float* ref_d, uint32_t count, Node* out_d, cudaStream_t s) {
  k_pack_nodes<<<grid_for(count, 256), 256, 0, s>>>(ref_d, count, out_d);
}

void launch_gather_tris(const float* pos_d, const uint32_t* idx_d, uint32_t tri_count, float4* out_d,
                        cudaStream_t s) {
  k_gather_tris<<<grid_for(tri_count, 256), 256, 0, s>>>(pos_d, idx_d, tri_count, out_d);
}

void launch_unpack(const Node* nodes, uint32_t count, const float4* tris, uint32_t tri_count, float* ref_d,
                   uint32_t* idx_d, cudaStream_t s) {
  k_unpack<<<grid_for(count > tri_count ? count : tri_count, 256), 256, 0, s>>>(nodes, count, tris, tri_count, ref_d,
                                                                                idx_d);
}

void launch_closest(const Node* nodes, uint32_t node_count, const float4* tris, const float* rays_d, uint32_t n,
                    double tMin, double tMax, int32_t* prim, float* t, float* u, float* v, uint32_t* queue,
                    uint32_t* ctr, bool exact_only, bool top_levels, cudaStream_t s, const Node* wide,
                    const NearTree* near) {
  if (n == 0) return;
  const ApiPolicy P{rays_d, n, tris, prim, t, u, v, tMin};
  using Listed = Queued<ApiPolicy>;
  TravArgs A{nodes, node_count, tris, tMin, tMax, queue, ctr + 1, ctr + 2, ctr, nullptr, top_levels ? 1 : 0};
  if (exact_only) {
    TravArgs E = A;
    E.queue = nullptr;
    k_closest_exact_t<ApiPolicy><<<grid_for(n, 128), 128, 0, s>>>(E, P);
    return;
  }
  static const int blocks = persistent_blocks((const void*)k_closest_fast_t<ApiPolicy>, ApiPolicy::kThreads);
  static const int wide_blocks = persistent_blocks((const void*)k_closest_wide_t<ApiPolicy>, ApiPolicy::kThreads);
  static const int near_blocks = persistent_blocks((const void*)k_closest_near_t<ApiPolicy>, ApiPolicy::kNearThreads);
  const int want = (int)((n + ApiPolicy::kThreads - 1) / ApiPolicy::kThreads);
  if (near) {
    TravArgs N = A;
    N.near = {(const Node*)near->records.ptr, tris, 0, near->bound, near->far};
    N.leaf_of = (const uint32_t*)near->leaf_of.ptr;
    k_closest_near_t<ApiPolicy><<<near_blocks, ApiPolicy::kNearThreads, 0, s>>>(N, P);
    // The rays it hands on, in the reference's order: over the four-wide view
    // where they may be many (`wide` is then given), else over the binary nodes.
    A.top_scenes = 0;
    A.work = ctr + 3;
    A.wide = wide;
    const Listed L{P, queue, ctr + 1};
    if (wide) {
      A.queue = queue + n;
      A.queue_len = ctr + 4;
      launch_after(k_closest_wide_t<Listed>, want < wide_blocks ? want : wide_blocks, ApiPolicy::kThreads, 0, s, A, L);
      launch_after(k_closest_exact_t<Listed>, grid_for(n < 4096 ? n : 4096, 128), 128, 0, s, A, L);
    } else {
      k_closest_fast_t<Listed, true><<<want < blocks ? want : blocks, ApiPolicy::kThreads, 0, s>>>(A, L);
    }
  } else {
    if (wide) {
      A.wide = wide;
      A.top_scenes = 0;
      k_closest_wide_t<ApiPolicy><<<want < wide_blocks ? want : wide_blocks, ApiPolicy::kThreads, 0, s>>>(A, P);
    } else {
      k_closest_fast_t<ApiPolicy><<<want < blocks ? want : blocks, ApiPolicy::kThreads, top_smem_bytes(A.top_scenes), s>>>(A, P);
    }
    // Slow path over the rays the fast kernel queued (length read on the device).
    k_closest_exact_t<ApiPolicy><<<grid_for(n < 4096 ? n : 4096, 128), 128, 0, s>>>(A, P);
  }
  launch_after(k_refine_api, grid_for(n, 256), 256, 0, s, P);
}

void launch_wide_view(const Node* nodes, uint32_t node_count, Node* wide, cudaStream_t s) {
  launch_build_wide(nodes, node_count, wide, s);
}

void launch_pick(const Node* nodes, uint32_t node_count, const float4* tris, const double* rays, bool on_device,
                 uint32_t n, double tMin, double tMax, PickHit* out_d, cudaStream_t s) {
  if (n == 0) return;
  TravArgs A{nodes, node_count, tris, tMin, tMax, nullptr, nullptr, nullptr, nullptr};
  if (on_device) {
    k_pick<<<n, 32, 0, s>>>(A, PickArray{rays}, out_d);
  } else {
    PickArgs args{};
    for (uint32_t i = 0; i < n * 6 && i < kPickArgs * 6; i++) args.r[i] = rays[i];
    k_pick<<<n < kPickArgs ? n : kPickArgs, 32, 0, s>>>(A, args, out_d);
  }
}

void launch_closest_d(const Node* nodes, uint32_t node_count, const float4* tris, const double* rays_d, uint32_t n,
                      double tMin, double tMax, int32_t* prim, double* t, double* u, double* v, unsigned* err,
                      cudaStream_t s) {
  if (n == 0) return;
  TravArgs A{nodes, node_count, tris, tMin, tMax, nullptr, nullptr, nullptr, err};
  k_closest_exact_d<<<grid_for(n, 128), 128, 0, s>>>(A, rays_d, n, prim, t, u, v);
}

}  // namespace lucent
