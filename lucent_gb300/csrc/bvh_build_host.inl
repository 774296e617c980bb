// Host orchestration of the GPU BVH builder (included by bvh_build.cu).
#include <algorithm>

#include "api_util.h"

namespace lucent {

// Writes to every page of a host buffer that a copy from the device is about to
// fill: a copy into pages that were never touched faults them one by one from
// the device's side (6 MB into a fresh allocation: 6 ms; touched first, 0.2).
static void touch_pages(void* p, size_t bytes) {
  for (size_t i = 0; i < bytes; i += 4096) ((volatile char*)p)[i] = 0;
  if (bytes) ((volatile char*)p)[bytes - 1] = 0;
}

// Builds the BVH of `n` triangles at `pos_d` (device, 9 floats each); `out`
// says what is wanted. Before this form (a launch per step and level with the
// host reading each level's nodes, one warp walking each small node out of L2,
// the tree renumbered on the host): 2,503 triangles 0.75 ms, 300,000 8.7 ms,
// 2,000,000 42 ms.
lucent_status gpu_build_bvh(const float* pos_d, uint32_t n, int max_leaf, int bins, cudaStream_t s, BuildOut& out) {
  using namespace build;
  if (bins < 2 || bins > kMaxBins) return fail(LUCENT_ERR_UNSUPPORTED, "bins must be in [2, %d]", kMaxBins);
  if (max_leaf < 1) return fail(LUCENT_ERR_INVALID, "maxLeafSize must be >= 1");
  if (n > (1u << 23)) return fail(LUCENT_ERR_UNSUPPORTED, "%u triangles; the limit is 2^23", n);
  lucent_status st = LUCENT_OK;
  if (n == 0) {  // bvh.ts:143-147
    for (int k = 0; k < 6; k++) out.bounds[k] = 0;
    for (int k = 0; k < 8 && out.nodes_host; k++) out.nodes_host[k] = 0.f;
    out.node_count = 1;
    out.depth = 0;
    if (out.nodes) {
      if ((st = out.nodes->reserve(sizeof(Node)))) return st;
      cudaError_t e = cudaMemsetAsync(out.nodes->ptr, 0, sizeof(Node), s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return cuda_fail(e, "empty BVH");
    }
    if (out.tris && (st = out.tris->reserve(48))) return st;
    if (out.order && (st = out.order->reserve(16))) return st;
    return LUCENT_OK;
  }

  // Scratch, one allocation. Big nodes hold more than sub_n triangles, so a
  // level has at most n / (sub_n + 1) of them, each with one ragged chunk.
  // Small builds: all big levels in one cluster. Whole builds of a soup, by
  // launches with subtrees of 1,024 and so: 2,503 triangles 435 and 316 us,
  // 8,000 569 and 427; 16,000, with blocks of 256 threads, 663 and 617 but of a
  // knot 672 and 683. Subtrees of 256 and 512 triangles: 2,503 321 and 322 us,
  // 4,000 373 and 393, 12,000 548 and 519; of 128, 2,503 takes 346.
  const bool clustered = n <= 12288;
  const uint32_t sub_n = !clustered ? kSub : n <= 4096 ? 256 : 512;
  const uint32_t nrec = 2 * n - 1, big_cap = n / (sub_n + 1) + 1, chunk_cap = n / kChunk + big_cap;
  const size_t words = (size_t)3 * bins * 7;
  struct Part {
    size_t bytes;
    void* ptr;
  };
  Part b_lo{(size_t)n * 16}, b_hi{(size_t)n * 16}, b_cz{(size_t)n * 4}, b_tri0{(size_t)n * 4}, b_tri1{(size_t)n * 4},
      b_tri2{(size_t)n * 4}, b_P{(size_t)n * 4}, b_Q{(size_t)n * 4}, b_recs{(size_t)nrec * 32},
      b_parent{(size_t)nrec * 4}, b_arrived{(size_t)nrec * 4}, b_inner{(size_t)nrec * 4}, b_height{(size_t)nrec * 4},
      b_ctr{kCtrBuild * 4}, b_small{(size_t)n * sizeof(Task)}, b_bins{big_cap * words * 4},
      b_bits{(size_t)chunk_cap * kChunk / 8}, b_count{(size_t)chunk_cap * sizeof(uint2)};
  Part b_big[2], b_box[2], b_chunk[2];
  TempBuffer scratch, ref;
  {
    for (int k = 0; k < 2; k++) {
      b_big[k].bytes = (size_t)big_cap * sizeof(Big);
      b_box[k].bytes = (size_t)big_cap * 48;
      b_chunk[k].bytes = (size_t)chunk_cap * sizeof(Chunk);
    }
    Part* all[] = {&b_lo, &b_hi, &b_cz, &b_tri0, &b_tri1, &b_tri2, &b_P, &b_Q, &b_recs, &b_parent, &b_arrived, &b_inner,
                   &b_height, &b_ctr, &b_small, &b_bins, &b_bits, &b_count, &b_big[0], &b_big[1], &b_box[0], &b_box[1],
                   &b_chunk[0], &b_chunk[1]};
    size_t total = 0;
    for (Part* p : all) total += (p->bytes + 255) & ~(size_t)255;
    if ((st = scratch.reserve(total, s))) return st;
    char* at = (char*)scratch.ptr;
    for (Part* p : all) {
      p->ptr = at;
      at += (p->bytes + 255) & ~(size_t)255;
    }
  }
  auto done = [&](lucent_status code) {
    ref.release();
    scratch.release();
    return code;
  };
#define BB_CUDA(x, what)                                      \
  do {                                                        \
    cudaError_t e_ = (x);                                     \
    if (e_ != cudaSuccess) return done(cuda_fail(e_, what));  \
  } while (0)

  Ctx cx;
  cx.p = {(const float4*)b_lo.ptr, (const float4*)b_hi.ptr, (const float*)b_cz.ptr};
  cx.tri[0] = (uint32_t*)b_tri0.ptr;
  cx.tri[1] = (uint32_t*)b_tri1.ptr;
  cx.tri[2] = (uint32_t*)b_tri2.ptr;
  cx.recs = (float4*)b_recs.ptr;
  cx.parent = (uint32_t*)b_parent.ptr;
  cx.ctr = (uint32_t*)b_ctr.ptr;
  cx.small = (Task*)b_small.ptr;
  for (int k = 0; k < 2; k++) {
    cx.big[k] = (Big*)b_big[k].ptr;
    cx.box[k] = (unsigned*)b_box[k].ptr;
    cx.chunk[k] = (Chunk*)b_chunk[k].ptr;
  }
  cx.bins = (unsigned*)b_bins.ptr;
  cx.bits = (unsigned*)b_bits.ptr;
  cx.count = (uint2*)b_count.ptr;
  cx.P = (int32_t*)b_P.ptr;
  cx.Q = (int32_t*)b_Q.ptr;
  cx.n = n;
  cx.big_cap = big_cap;
  cx.chunk_cap = chunk_cap;
  cx.rec_cap = nrec;
  cx.sub = sub_n;
  cx.max_leaf = max_leaf;
  cx.nbins = bins;

  BB_CUDA(cudaMemsetAsync(cx.ctr, 0, kCtrBuild * 4, s), "clear counters");
  BB_CUDA(cudaMemsetAsync(cx.recs, 0xff, (size_t)nrec * 32, s), "clear nodes");
  BB_CUDA(cudaMemsetAsync(cx.parent, 0, (char*)b_height.ptr + b_height.bytes - (char*)b_parent.ptr, s), "clear tree");
  k_init<<<1, 32, 0, s>>>(cx);
  launch_after(k_prim_bounds, std::min<uint32_t>((n + 255) / 256, 152 * 8), 256, 0, s, pos_d, cx, (float4*)b_lo.ptr,
               (float4*)b_hi.ptr, (float*)b_cz.ptr);
  uint32_t got[kCtrBuild] = {0};
  int p = 0;
  uint32_t small = 0;  // blocks of the subtree kernel
  if (n > sub_n) {
    launch_after(k_clear_bins, std::min<uint32_t>((uint32_t)(big_cap * words + 255) / 256, 152 * 8), 256, 0, s, cx.bins,
                 big_cap * words);
    // Two levels more than halving would take, then a few at a time until no
    // big node is left; a level of no nodes costs five empty launches.
    int levels = 3;
    while ((n >> (levels - 2)) > (uint32_t)kSub) levels++;
    for (int total = 0; !clustered; levels = 3) {
      if ((total += levels) > 8192) return done(fail(LUCENT_ERR_DEVICE, "BVH build did not converge"));
      for (int k = 0; k < levels; k++, p ^= 1) {
        launch_after(k_big_bins, chunk_cap, 256, words * 4, s, cx, p);
        launch_after(k_big_sah, (big_cap + 3) / 4, 128, 4 * words * 4, s, cx, p);
        launch_after(k_big_count, chunk_cap, 256, 0, s, cx, p);
        launch_after(k_big_place, chunk_cap, 256, 0, s, cx, p);
        launch_after(k_big_move, chunk_cap, 256, 0, s, cx, p);
      }
      BB_CUDA(cudaMemcpyAsync(got, cx.ctr, sizeof got, cudaMemcpyDeviceToHost, s), "read counters");
      BB_CUDA(cudaStreamSynchronize(s), "big levels");
      if (got[kErrW]) return done(fail(LUCENT_ERR_DEVICE, "BVH build raised device error 0x%x", got[kErrW]));
      if (got[kNBig + p] == 0) break;
    }
    small = got[kNSmall];
    if (clustered) {
      launch_after(k_big_levels, kCluster, kLevelThreads, kLevelThreads / 32 * words * 4, s, cx);
      small = std::min(n, 2 * 152u);  // the device knows how many there are
    }
  } else {
    small = 1;
  }
  if (small > n) return done(fail(LUCENT_ERR_DEVICE, "task list overflow"));
  // Subtrees that all run at once take 16 warps each, as the launch lasts as
  // long as one of them (82,000 triangles, whole build: 651 us against 703 with
  // 8); more of them 8 (2,000,000: 3.80 ms against 3.94). Subtrees of 512 or
  // 2,048 triangles measured slower after big levels by launches.
  const int threads = small <= 3 * 152 ? kSubThreads : kSubThreads / 2;
  const size_t smem = sub_bytes(sub_n, bins, threads);
  // The most any build asks for, so that builds on several threads agree.
  BB_CUDA(cudaFuncSetAttribute((const void*)k_subtree, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)sub_bytes(kSub, kMaxBins, kSubThreads)),
          "shared memory of the subtree kernel");
  if (small) launch_after(k_subtree, small, threads, smem, s, cx);
  const int g = (int)((nrec + 127) / 128);
  uint32_t* inner = (uint32_t*)b_inner.ptr;
  uint32_t* height = (uint32_t*)b_height.ptr;
  launch_after(k_tree_counts, g, 128, 0, s, cx, (uint32_t*)b_arrived.ptr, inner, height, nrec);
  uint32_t root[2];
  float box[8];
  BB_CUDA(cudaMemcpyAsync(got, cx.ctr, sizeof got, cudaMemcpyDeviceToHost, s), "read counters");
  BB_CUDA(cudaMemcpyAsync(&root[0], inner, 4, cudaMemcpyDeviceToHost, s), "read node count");
  BB_CUDA(cudaMemcpyAsync(&root[1], height, 4, cudaMemcpyDeviceToHost, s), "read depth");
  BB_CUDA(cudaMemcpyAsync(box, cx.recs, 32, cudaMemcpyDeviceToHost, s), "read root");
  BB_CUDA(cudaStreamSynchronize(s), "build");
  if (got[kErrW]) return done(fail(LUCENT_ERR_DEVICE, "BVH build raised device error 0x%x", got[kErrW]));
  const uint32_t nr = 2 * root[0] + 1;
  if (nr > nrec) return done(fail(LUCENT_ERR_DEVICE, "BVH build produced %u nodes", nr));
  out.node_count = nr;
  out.depth = root[1];
  for (int k = 0; k < 3; k++) {  // bvh.ts:245-251: measure(0, triCount) = the root's box
    out.bounds[k] = box[k];
    out.bounds[3 + k] = box[4 + k];
  }
  if ((out.nodes && (st = out.nodes->reserve((size_t)nr * sizeof(Node)))) ||
      (out.tris && (st = out.tris->reserve((size_t)n * 48))) || (out.order && (st = out.order->reserve((size_t)n * 4))) ||
      (out.nodes_host && (st = ref.reserve((size_t)nr * 32, s))))
    return done(st);
  k_tree_emit<<<g, 128, 0, s>>>(cx, inner, nrec, out.nodes ? (float4*)out.nodes->ptr : nullptr, (float4*)ref.ptr);
  if (out.tris) launch_gather_tris(pos_d, cx.tri[2], n, (float4*)out.tris->ptr, s);
  if (out.order)
    BB_CUDA(cudaMemcpyAsync(out.order->ptr, cx.tri[2], (size_t)n * 4, cudaMemcpyDeviceToDevice, s), "copy order");
  BB_CUDA(cudaGetLastError(), "build kernels");
  if (out.nodes_host) touch_pages(out.nodes_host, (size_t)nr * 32);
  if (out.tri_host) touch_pages(out.tri_host, (size_t)n * 4);
  if (out.nodes_host)
    BB_CUDA(cudaMemcpyAsync(out.nodes_host, ref.ptr, (size_t)nr * 32, cudaMemcpyDeviceToHost, s), "read nodes");
  if (out.tri_host)
    BB_CUDA(cudaMemcpyAsync(out.tri_host, cx.tri[2], (size_t)n * 4, cudaMemcpyDeviceToHost, s), "read triIndices");
  BB_CUDA(cudaStreamSynchronize(s), "pack built BVH");
  return done(LUCENT_OK);
#undef BB_CUDA
}

}  // namespace lucent
