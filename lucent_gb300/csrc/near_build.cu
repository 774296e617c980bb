// The nearest-first traversal's view of a tree (traverse_near.cuh): leaf boxes
// grown by the rounding error of the reference's triangle test, their unions
// above, four grandchildren per record group, and each slot's leaf.
#include <cmath>
#include <cstring>

#include "api_util.h"
#include "internal.h"
#include "near_growth.h"
#include "traverse_near.cuh"

namespace lucent {
namespace {

enum : int { kNearBad = 0, kNearBig = 1, kNearRise = 2, kNearWords = 3 };

// Parents, and the checks that the traversal's argument needs: one parent per
// node (k_near_leaves sees to it that there is one), child boxes inside their
// parent's, leaves the reference can hold.
__global__ void k_near_parents(const Node* __restrict__ nodes, uint32_t n_nodes, uint32_t* __restrict__ parent,
                               uint32_t* __restrict__ words) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  const Node nd = load_node(nodes, n);
  const int cnt = node_count(nd), f = node_first(nd);
  bool ok = cnt <= kNearMaxLeaf;
  if (cnt == 0) {
    for (int k = f; k <= f + 1; k++) {
      const Node ch = load_node(nodes, k);
      ok = ok && ch.lo.x >= nd.lo.x && ch.lo.y >= nd.lo.y && ch.lo.z >= nd.lo.z && ch.hi.x <= nd.hi.x &&
           ch.hi.y <= nd.hi.y && ch.hi.z <= nd.hi.z;
      ok = atomicExch(parent + k, n + 1) == 0 && ok;
    }
  }
  if (!ok) atomicOr(words + kNearBad, 1u);
}

// Leaves: grown box, slots' leaf; then upwards, the second child to arrive at
// a node writing the union (a node's writer stops or goes on to its parent, a
// lower index, so every climb ends). Bound by that chain: what the next level
// needs is loaded before the level's atomic, which orders the boxes by itself
// (before: two fences a level, and one atomic a leaf on the word of the largest
// rise). 20,480 and 300,000 triangles: 37 and 88 us before, 26 and 40 now.
__global__ void k_near_leaves(const Node* __restrict__ nodes, uint32_t n_nodes, const float4* __restrict__ tris,
                              float diag, const uint32_t* __restrict__ parent, uint32_t* __restrict__ arrived,
                              Node* cull, uint32_t* tail, uint32_t* __restrict__ leaf_of, uint32_t* words) {
  wait_for_previous();
  uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  if (n > 0 && parent[n] == 0) {
    // Outside the tree (children have higher indices than their parent, so all
    // that has one hangs below the root or below such a node): none of its
    // boxes bounds what the reference visits, but a leaf would claim its slots.
    atomicOr(words + kNearBad, 1u);
    return;
  }
  const Node nd = load_node(nodes, n);
  const int cnt = node_count(nd), f = node_first(nd);
  if (cnt == 0) return;
  float g = 0.f, rise = 0.f;
  bool ok = true;
  for (int k = 0; k < cnt; k++) {
    const size_t s = (size_t)(f + k);
    const float4 v[3] = {__ldg(tris + 3 * s), __ldg(tris + 3 * s + 1), __ldg(tris + 3 * s + 2)};
    g = fmaxf(g, leaf_growth(v[0], v[1], v[2], 2.5f * diag, rise));
    for (int j = 0; j < 3; j++)
      ok = ok && v[j].x >= nd.lo.x && v[j].y >= nd.lo.y && v[j].z >= nd.lo.z && v[j].x <= nd.hi.x &&
           v[j].y <= nd.hi.y && v[j].z <= nd.hi.z;
    leaf_of[s] = n;
  }
  if (!ok) atomicOr(words + kNearBad, 1u);
  if (g > diag * 0.03125f) atomicAdd(words + kNearBig, 1u);
  const unsigned act = __activemask();
  const unsigned most = __reduce_max_sync(act, __float_as_uint(rise));  // positive floats order as integers
  if ((int)(threadIdx.x & 31) == __ffs(act) - 1 && most > __ldcg(words + kNearRise)) atomicMax(words + kNearRise, most);
  Node c;
  c.lo = make_float4(__fsub_rd(nd.lo.x, g), __fsub_rd(nd.lo.y, g), __fsub_rd(nd.lo.z, g),
                     __int_as_float(kNearLeaf | f << 8 | (cnt & kNearMaxLeaf)));
  c.hi = make_float4(__fadd_ru(nd.hi.x, g), __fadd_ru(nd.hi.y, g), __fadd_ru(nd.hi.z, g), __int_as_float(f));
  uint32_t end = (uint32_t)(f + cnt), up = parent[n];
  while (true) {  // (hi.w and `tail`: the subtree's slots, which have to be in the order the reference visits them)
    float4* p = reinterpret_cast<float4*>(cull) + 2 * (size_t)n;
    __stcg(p, c.lo);
    __stcg(p + 1, c.hi);
    __stcg(tail + n, end);
    if (up == 0) return;
    n = up - 1;
    const int first = node_first(load_node(nodes, n));
    up = parent[n];
    if (arrive(arrived + n) == 0) return;  // the sibling comes later
    const float4* q = reinterpret_cast<const float4*>(cull) + 2 * (size_t)first;
    const float4 al = __ldcg(q), ah = __ldcg(q + 1), bl = __ldcg(q + 2), bh = __ldcg(q + 3);
    c.lo = make_float4(fminf(al.x, bl.x), fminf(al.y, bl.y), fminf(al.z, bl.z), __int_as_float((int)n));
    c.hi = make_float4(fmaxf(ah.x, bh.x), fmaxf(ah.y, bh.y), fmaxf(ah.z, bh.z), ah.w);
    end = __ldcg(tail + first + 1);
    if (__ldcg(tail + first) > (uint32_t)__float_as_int(bh.w)) atomicOr(words + kNearBad, 1u);
  }
}

// Records 4 n .. 4 n + 3 of every inner node n (and of a tree that is one
// leaf, that leaf as record 0).
__global__ void k_near_records(const Node* __restrict__ nodes, const Node* __restrict__ cull, uint32_t n_nodes,
                               Node* __restrict__ out) {
  wait_for_previous();
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  const Node nd = load_node(nodes, n);
  if (node_count(nd) > 0 && n > 0) return;  // never expanded
  const float inf = __int_as_float(0x7f800000);
  Node rec[kWide];
#pragma unroll
  for (int k = 0; k < kWide; k++)  // unused: an inverted box, a leaf of no triangles
    rec[k] = {make_float4(inf, inf, inf, __int_as_float(kNearNone)), make_float4(-inf, -inf, -inf, 0.f)};
  if (node_count(nd) > 0) {
    rec[0] = load_node(cull, n);
  } else {
    const int f = node_first(nd);
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const Node ch = load_node(nodes, f + c);
      if (node_count(ch) > 0) {
        rec[2 * c] = load_node(cull, f + c);
      } else {
        const int g = node_first(ch);
        rec[2 * c] = load_node(cull, g);
        rec[2 * c + 1] = load_node(cull, g + 1);
      }
    }
  }
  float4* o = reinterpret_cast<float4*>(out + (size_t)kWide * n);
#pragma unroll
  for (int k = 0; k < kWide; k++) {
    o[2 * k] = rec[k].lo;
    o[2 * k + 1] = rec[k].hi;
  }
}

}  // namespace

lucent_status build_near_view(const Node* nodes, uint32_t n_nodes, const float4* tris, uint32_t n_tris,
                              const float lo[3], const float hi[3], NearTree& out, cudaStream_t s) {
  out.usable = false;
  if (n_nodes == 0 || n_tris == 0) return LUCENT_OK;
  double d2 = 0;
  float c[3];
  for (int k = 0; k < 3; k++) {
    c[k] = 0.5f * lo[k] + 0.5f * hi[k];
    d2 += ((double)hi[k] - lo[k]) * ((double)hi[k] - lo[k]);
  }
  const float diag = (float)(sqrt(d2) * 1.000001);
  if (!(diag > 1e-15f) || !(diag < 1e9f)) return LUCENT_OK;
  const float mag = fmaxf(fmaxf(fabsf(c[0]), fabsf(c[1])), fabsf(c[2]));
  if (!(mag < 1e3f * diag)) return LUCENT_OK;
  lucent_status st;
  TempBuffer tmp;
  const size_t cull = (size_t)n_nodes * sizeof(Node), idx = (size_t)n_nodes * 4;
  if ((st = out.records.reserve((size_t)n_nodes * kWide * sizeof(Node))) ||
      (st = out.leaf_of.reserve((size_t)n_tris * 4)) || (st = tmp.reserve(cull + 3 * idx + 64, s))) {
    out.release();
    if (st != LUCENT_ERR_OOM) return st;
    cudaGetLastError();  // no room for it: not usable, and nothing else is wrong
    clear_error();
    return LUCENT_OK;
  }
  char* b = (char*)tmp.ptr;
  uint32_t* parent = (uint32_t*)(b + cull);
  uint32_t* arrived = parent + n_nodes;
  uint32_t* words = arrived + n_nodes;
  uint32_t* tail = words + 16;
  uint32_t got[kNearWords] = {1, 0, 0};
  const int g = (int)((n_nodes + 127) / 128);
  cudaError_t e = cudaMemsetAsync(parent, 0, 2 * idx + kNearWords * 4, s);
  if (e == cudaSuccess) {
    k_near_parents<<<g, 128, 0, s>>>(nodes, n_nodes, parent, words);
    launch_after(k_near_leaves, g, 128, 0, s, nodes, n_nodes, tris, diag, parent, arrived, (Node*)b, tail,
                 (uint32_t*)out.leaf_of.ptr, words);
    launch_after(k_near_records, g, 128, 0, s, nodes, (const Node*)b, n_nodes, (Node*)out.records.ptr);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(got, words, sizeof got, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  tmp.release();
  if (e != cudaSuccess) return cuda_fail(e, "nearest-first view");
  out.usable = got[kNearBad] == 0 && got[kNearBig] <= 64;
  // Origins beyond two diagonals (less the rounding of centre and distance)
  // grow every box of the ray's traversal by `rise` per unit. That pays while
  // it stays under a tenth of a leaf (about diag / sqrt(n) for a surface):
  // meshes reach some ten to hundred diagonals, a fine mesh beside a large
  // tilted triangle little more than two.
  float rise;
  memcpy(&rise, &got[kNearRise], 4);
  const float extra = 0.1f * diag / sqrtf((float)n_tris) / fmaxf(rise, 1e-30f);
  out.far = make_float2(1.99f * diag, rise);
  out.bound = make_float4(c[0], c[1], c[2], fminf(1.99f * diag + extra, 1e4f * diag));
  out.wide_range = out.bound.w >= 64.f * diag;
  if (!out.usable) out.release();
  return LUCENT_OK;
}

}  // namespace lucent
