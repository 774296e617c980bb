// C ABI: status codes, thread-local error text, BVH handle for closest-hit.
#include <cmath>
#include <cstring>
#include <cstdarg>
#include <cstdio>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/lucent.h"
#include "api_util.h"
#include "internal.h"

using namespace lucent;

namespace lucent {

static thread_local std::string g_last_error;

lucent_status fail(lucent_status code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}

void clear_error() { g_last_error.clear(); }

lucent_status cuda_fail(cudaError_t e, const char* what) {
  cudaGetLastError();  // clear the sticky-free error state
  if (e == cudaErrorMemoryAllocation) return fail(LUCENT_ERR_OOM, "%s: %s", what, cudaGetErrorString(e));
  return fail(LUCENT_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

uint64_t first_not_finite(const float* v, uint64_t n) {
  // A block's exponents at a time, without a branch per value (vectorised by
  // the compiler): 2.7 M floats 1.9 -> 0.3 ms on a Grace core.
  constexpr uint64_t kBlock = 4096;
  for (uint64_t b = 0; b < n; b += kBlock) {
    const uint64_t e = b + kBlock < n ? b + kBlock : n;
    uint32_t bad = 0;
    for (uint64_t i = b; i < e; i++) {
      uint32_t w;
      memcpy(&w, v + i, 4);
      bad |= (w & 0x7f800000u) == 0x7f800000u;
    }
    if (bad)
      for (uint64_t i = b; i < e; i++)
        if (!std::isfinite(v[i])) return i;
  }
  return n;
}

// The pool of a device for the memory of single calls and of BVH handles:
// cudaMalloc and cudaFree of a build's buffers cost as much as a small
// build (the last cudaFree of a 2 MiB block alone some 180 us). Stream-ordered,
// so threads and streams share it safely; it holds at most 1 GiB between calls
// (the driver takes back what is free beyond that), and gives what is free
// back when an ordinary allocation fails and on lucent_trim. 1 GiB holds the
// scratch of 6,000,000 triangles (168 bytes each): builds of so many take 12.8
// ms one after another, of 8,388,608, which map the rest anew each time, 20.1
// (of which that is some 2). `stream`: the pool's own, for allocations that
// outlive a call.
struct Pool {
  int device = 0;
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;
  std::mutex lock;
  std::vector<void*> waiting;  // of closed handles, until the device can be waited for
  void give_waiting_back();
};
static Pool* device_pool() {  // of the current device
  static std::mutex lock;
  static Pool* const pools = new Pool[64];  // never destroyed: handles may outlive any static object
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> hold(lock);
  Pool& P = pools[dev];
  if (!P.pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaStream_t stream;
    if (cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    if (cudaMemPoolCreate(&P.pool, &props) != cudaSuccess) {
      cudaStreamDestroy(stream);
      P.pool = nullptr;
      return nullptr;
    }
    uint64_t keep = 1ull << 30;
    cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    P.device = dev;
    P.stream = stream;
  }
  return &P;
}

std::shared_mutex& capture_lock() {
  static std::shared_mutex* const m = new std::shared_mutex;
  return *m;
}

// Blocks that no event stands for are given back once their device has been
// waited for, as cudaFree would; where that is refused, they stay for the next time.
void Pool::give_waiting_back() {
  std::lock_guard<std::mutex> hold(lock);
  if (waiting.empty()) return;
  std::unique_lock<std::shared_mutex> no_capture(capture_lock(), std::try_to_lock);
  if (!no_capture) return;
  int before = 0;
  cudaError_t e = cudaGetDevice(&before);
  if (e == cudaSuccess && before != device) e = cudaSetDevice(device);
  if (e == cudaSuccess) {
    e = cudaDeviceSynchronize();
    if (before != device) cudaSetDevice(before);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  for (void* p : waiting) cudaFreeAsync(p, stream);
  waiting.clear();
}

lucent_status StreamUses::begin(cudaStream_t s) {
  unsigned long long id = 0;
  if (cudaError_t e = cudaStreamGetId(s, &id); e != cudaSuccess) return cuda_fail(e, "stream");
  for (size_t k = 0; k < uses.size(); k++)
    if (uses[k].stream == id) {
      std::swap(uses[k], uses.back());
      return LUCENT_OK;
    }
  if (uses.size() < 4) {
    cudaEvent_t event;
    if (cudaError_t e = cudaEventCreateWithFlags(&event, cudaEventDisableTiming); e != cudaSuccess)
      return cuda_fail(e, "event");
    uses.push_back({id, event, false});
  } else {
    Use& u = uses.front();
    if (u.open && cudaStreamWaitEvent(home->stream, u.event, 0) != cudaSuccess) {
      cudaGetLastError();
      unordered = true;
    }
    u.stream = id;
    u.open = false;
    std::swap(u, uses.back());
  }
  return LUCENT_OK;
}

lucent_status StreamUses::end(cudaStream_t s) {
  uses.back().open = true;
  const cudaError_t e = cudaEventRecord(uses.back().event, s);
  if (e == cudaSuccess) return LUCENT_OK;
  unordered = true;
  return cuda_fail(e, "event");
}

void StreamUses::give_back(void* ptr, bool held) {
  if (!held && !unordered) {
    bool ok = true;
    for (Use& u : uses) {
      if (u.open) ok = cudaStreamWaitEvent(home->stream, u.event, 0) == cudaSuccess && ok;
      u.open = false;
    }
    if (ok && cudaFreeAsync(ptr, home->stream) == cudaSuccess) return;
    cudaGetLastError();
    unordered = true;
  }
  kept.push_back(ptr);
}

void StreamUses::close() {
  for (Use& u : uses) cudaEventDestroy(u.event);
  uses.clear();
  if (!home) return;
  {
    std::lock_guard<std::mutex> hold(home->lock);
    home->waiting.insert(home->waiting.end(), kept.begin(), kept.end());
  }
  kept.clear();
  home->give_waiting_back();
}

static void trim_pool(Pool& P) {
  P.give_waiting_back();
  cudaMemPoolTrimTo(P.pool, 0);
}

void trim_temporaries() {
  if (Pool* P = device_pool()) trim_pool(*P);
}

static lucent_status pool_alloc(void** ptr, size_t bytes, Pool* P, cudaStream_t s) {
  *ptr = nullptr;
  if (!P) return cuda_fail(cudaGetLastError(), "memory pool");
  cudaError_t e = cudaMallocFromPoolAsync(ptr, bytes, P->pool, s);
  if (e == cudaErrorMemoryAllocation) {  // once more without what the pool holds
    cudaGetLastError();
    trim_pool(*P);
    e = cudaMallocFromPoolAsync(ptr, bytes, P->pool, s);
  }
  if (e == cudaSuccess) return LUCENT_OK;
  *ptr = nullptr;
  return cuda_fail(e, "cudaMallocFromPoolAsync");
}

lucent_status TempBuffer::reserve(size_t bytes, cudaStream_t s) {
  release();
  stream = s;
  return pool_alloc(&ptr, bytes < 256 ? 256 : bytes, device_pool(), s);
}

void TempBuffer::release() {
  if (ptr) cudaFreeAsync(ptr, stream);
  ptr = nullptr;
}

lucent_status DeviceBuffer::reserve(size_t bytes) {
  if (bytes <= cap) return LUCENT_OK;
  release();
  const size_t want = bytes < 256 ? 256 : bytes;
  if (uses) {  // allocated on the pool's stream and waited for: usable on any stream
    if (!uses->home) uses->home = device_pool();
    Pool* const P = uses->home;
    if (lucent_status st = pool_alloc(&ptr, want, P, P ? P->stream : nullptr)) return st;
    if (cudaError_t e = cudaStreamSynchronize(P->stream); e != cudaSuccess) {
      cudaFreeAsync(ptr, P->stream);
      ptr = nullptr;
      return cuda_fail(e, "pool allocation");
    }
    cap = want;
    return LUCENT_OK;
  }
  cudaError_t e = cudaMalloc(&ptr, want);
  if (e == cudaErrorMemoryAllocation) {  // once more without what the pool holds
    cudaGetLastError();
    trim_temporaries();
    e = cudaMalloc(&ptr, want);
  }
  if (e != cudaSuccess) {
    ptr = nullptr;
    return cuda_fail(e, "cudaMalloc");
  }
  cap = want;
  return LUCENT_OK;
}

void DeviceBuffer::release() {
  if (ptr && uses)
    uses->give_back(ptr, held);
  else if (ptr)
    cudaFree(ptr);
  ptr = nullptr;
  cap = 0;
  held = false;
}

}  // namespace lucent

struct lucent_bvh {
  uint32_t node_count = 0, tri_count = 0;
  // Tree depth (root = 0). Trees whose depth could overflow the reference's
  // 64-entry stack take the all-binary64 path, which reproduces the overflow.
  uint32_t depth = 0;
  int mode = LUCENT_TRAVERSE_WIDE;
  StreamUses uses;
  // From the pool: with everything else pooled, a cudaMalloc of the scratch maps
  // a new 2 MiB block (100 us of a new tree's first query).
  DeviceBuffer nodes{nullptr, 0, &uses}, tris{nullptr, 0, &uses}, scratch{nullptr, 0, &uses}, stage{nullptr, 0, &uses};
  float lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};  // the root's box
  NearTree near{&uses};  // nearest-first view (LUCENT_TRAVERSE_WIDE, where usable), built on first use
  bool near_tried = false;
  DeviceBuffer wide{nullptr, 0, &uses};  // four-wide view of `nodes` (LUCENT_TRAVERSE_WIDE otherwise), built on first use
  bool views = false;  // what LUCENT_TRAVERSE_WIDE reads has been built, and is there for every stream
};

static void set_root(lucent_bvh* b, const float* nodes) {
  for (int k = 0; k < 3; k++) {
    b->lo[k] = nodes[k];
    b->hi[k] = nodes[4 + k];
  }
}

extern "C" {

const char* lucent_last_error(void) { return g_last_error.c_str(); }
int32_t lucent_version(void) { return 100; }

// Depth of a (validated) reference-layout tree; root = 0.
uint32_t tree_depth(const float* nodes, uint32_t node_count, uint32_t tri_count) {
  if (tri_count == 0 || node_count == 0) return 0;
  std::vector<std::pair<uint32_t, uint32_t>> st{{0u, 0u}};
  uint32_t depth = 0;
  while (!st.empty()) {
    const auto [n, d] = st.back();
    st.pop_back();
    depth = d > depth ? d : depth;
    const float* r = nodes + (size_t)n * 8;
    if (r[7] > 0) continue;
    const uint32_t l = (uint32_t)r[3];
    st.push_back({l, d + 1});
    st.push_back({l + 1, d + 1});
  }
  return depth;
}

// Validates the reference layout so that no kernel can read out of bounds:
// children inside the array, leaf ranges inside triIndices, indices in range.
lucent_status validate_bvh(const float* nodes, uint32_t node_count, const uint32_t* tri, uint32_t tri_count) {
  if (node_count == 0) return fail(LUCENT_ERR_INVALID, "BVH has no nodes");
  if (tri_count > (1u << 23)) return fail(LUCENT_ERR_UNSUPPORTED, "%u triangles; the limit is 2^23", tri_count);
  for (uint32_t i = 0; i < tri_count; i++)
    if (tri[i] >= tri_count) return fail(LUCENT_ERR_INVALID, "triIndices[%u] = %u out of range", i, tri[i]);
  if (tri_count == 0) return LUCENT_OK;
  for (uint32_t n = 0; n < node_count; n++) {
    const float* r = nodes + (size_t)n * 8;
    const float lf = r[3], cnt = r[7];
    if (!(lf >= 0) || !(cnt >= 0) || lf != std::floor(lf) || cnt != std::floor(cnt))
      return fail(LUCENT_ERR_INVALID, "node %u has a malformed leftFirst/count", n);
    if (cnt > 0) {
      if ((double)lf + cnt > tri_count) return fail(LUCENT_ERR_INVALID, "leaf %u range past triIndices", n);
    } else if ((double)lf + 1 >= node_count || lf <= n) {
      return fail(LUCENT_ERR_INVALID, "node %u children out of range", n);
    }
    for (int k : {0, 1, 2, 4, 5, 6})
      if (!std::isfinite(r[k])) return fail(LUCENT_ERR_INVALID, "node %u has a non-finite bound", n);
  }
  return LUCENT_OK;
}

lucent_status lucent_bvh_create(const float* nodes, uint32_t node_count, const uint32_t* tri_indices,
                                uint32_t tri_count, const float* positions, lucent_bvh** out) {
  clear_error();
  if (!out || !nodes || (tri_count && (!tri_indices || !positions)))
    return fail(LUCENT_ERR_INVALID, "null argument");
  *out = nullptr;
  lucent_status st = validate_bvh(nodes, node_count, tri_indices, tri_count);
  if (st) return st;
  lucent_bvh* b = new lucent_bvh();
  b->node_count = node_count;
  b->tri_count = tri_count;
  b->depth = tree_depth(nodes, node_count, tri_count);
  DeviceBuffer ref, pos, idx;
  cudaStream_t s = 0;
  auto cleanup = [&](lucent_status code) {
    ref.release();
    pos.release();
    idx.release();
    if (code) {
      b->uses.unordered = true;
      lucent_bvh_destroy(b);
    }
    return code;
  };
  if ((st = b->nodes.reserve((size_t)node_count * sizeof(Node)))) return cleanup(st);
  if ((st = b->tris.reserve((size_t)(tri_count ? tri_count : 1) * 48))) return cleanup(st);
  if ((st = ref.reserve((size_t)node_count * 32))) return cleanup(st);
  cudaError_t e = cudaMemcpyAsync(ref.ptr, nodes, (size_t)node_count * 32, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return cleanup(cuda_fail(e, "upload nodes"));
  launch_pack_nodes((const float*)ref.ptr, node_count, (Node*)b->nodes.ptr, s);
  if (tri_count) {
    if ((st = pos.reserve((size_t)tri_count * 36)) || (st = idx.reserve((size_t)tri_count * 4))) return cleanup(st);
    e = cudaMemcpyAsync(pos.ptr, positions, (size_t)tri_count * 36, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(idx.ptr, tri_indices, (size_t)tri_count * 4, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cleanup(cuda_fail(e, "upload triangles"));
    launch_gather_tris((const float*)pos.ptr, (const uint32_t*)idx.ptr, tri_count, (float4*)b->tris.ptr, s);
  }
  e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return cleanup(cuda_fail(e, "bvh upload kernels"));
  set_root(b, nodes);
  cleanup(LUCENT_OK);
  *out = b;
  return LUCENT_OK;
}

static lucent_status build_common(const float* pos_d, uint32_t n, const lucent_bvh_opts* opts, cudaStream_t s,
                                  float* nodes_out, uint32_t* node_count_out, uint32_t* tri_out, double* bounds_out,
                                  lucent_bvh** handle_out) {
  const int max_leaf = opts ? (int)opts->max_leaf_size : 4;  // bvh.ts:33 defaults
  const int bins = opts ? (int)opts->bins : 12;
  lucent_bvh* b = handle_out ? new lucent_bvh() : nullptr;
  BuildOut out;
  if (b) {
    out.nodes = &b->nodes;
    out.tris = &b->tris;
  }
  out.nodes_host = nodes_out;
  out.tri_host = tri_out;
  lucent_status st = gpu_build_bvh(pos_d, n, max_leaf, bins, s, out);
  if (st) {
    if (b) b->uses.unordered = true;
    lucent_bvh_destroy(b);
    return st;
  }
  if (node_count_out) *node_count_out = out.node_count;
  if (bounds_out) memcpy(bounds_out, out.bounds, sizeof out.bounds);
  if (b) {
    b->node_count = out.node_count;
    b->tri_count = n;
    b->depth = out.depth;
    for (int k = 0; k < 3; k++) {
      b->lo[k] = (float)out.bounds[k];
      b->hi[k] = (float)out.bounds[3 + k];
    }
    *handle_out = b;
  }
  return LUCENT_OK;
}

lucent_status lucent_bvh_build(const float* positions, uint64_t n_floats, const lucent_bvh_opts* opts,
                               float* nodes_out, uint32_t* node_count_out, uint32_t* tri_indices_out,
                               double* bounds_out, lucent_bvh** handle_out, void* stream) {
  clear_error();
  if (handle_out) *handle_out = nullptr;
  if (n_floats % 9 != 0)  // bvh.ts:55-57
    return fail(LUCENT_ERR_INVALID, "positions length %llu is not a multiple of 9", (unsigned long long)n_floats);
  if (n_floats && !positions) return fail(LUCENT_ERR_INVALID, "null positions");
  const uint64_t n = n_floats / 9;
  if (n > (1u << 23)) return fail(LUCENT_ERR_UNSUPPORTED, "%llu triangles; the limit is 2^23", (unsigned long long)n);
  if (const uint64_t i = first_not_finite(positions, n_floats); i < n_floats)
    return fail(LUCENT_ERR_UNSUPPORTED, "positions[%llu] is not finite", (unsigned long long)i);
  cudaStream_t s = (cudaStream_t)stream;
  TempBuffer pos;
  lucent_status st = pos.reserve(n_floats * 4 + 4, s);
  if (st) return st;
  cudaError_t e = cudaMemcpyAsync(pos.ptr, positions, n_floats * 4, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) {
    pos.release();
    return cuda_fail(e, "upload positions");
  }
  st = build_common((const float*)pos.ptr, (uint32_t)n, opts, s, nodes_out, node_count_out, tri_indices_out,
                    bounds_out, handle_out);
  cudaStreamSynchronize(s);
  pos.release();
  return st;
}

lucent_status lucent_bvh_build_device(const float* positions_d, uint32_t tri_count, const lucent_bvh_opts* opts,
                                      lucent_bvh** handle_out, void* stream) {
  clear_error();
  if (!handle_out || (tri_count && !positions_d)) return fail(LUCENT_ERR_INVALID, "null argument");
  *handle_out = nullptr;
  return build_common(positions_d, tri_count, opts, (cudaStream_t)stream, nullptr, nullptr, nullptr, nullptr,
                      handle_out);
}

lucent_status lucent_trim(void) {
  clear_error();
  const cudaError_t e = cudaDeviceSynchronize();  // what is freed on a stream is free once the stream gets there
  if (e != cudaSuccess) return cuda_fail(e, "synchronize");
  trim_temporaries();
  return LUCENT_OK;
}

void lucent_bvh_destroy(lucent_bvh* b) {
  if (!b) return;
  b->nodes.release();
  b->tris.release();
  b->scratch.release();
  b->stage.release();
  b->wide.release();
  b->near.release();
  b->uses.close();
  delete b;
}

lucent_status lucent_bvh_info(const lucent_bvh* b, uint32_t* node_count, uint32_t* tri_count) {
  clear_error();
  if (!b) return fail(LUCENT_ERR_INVALID, "null bvh");
  if (node_count) *node_count = b->node_count;
  if (tri_count) *tri_count = b->tri_count;
  return LUCENT_OK;
}

lucent_status lucent_bvh_download(const lucent_bvh* b, float* nodes_out, uint32_t* tri_indices_out) {
  clear_error();
  if (!b || !nodes_out || (b->tri_count && !tri_indices_out)) return fail(LUCENT_ERR_INVALID, "null argument");
  DeviceBuffer tmp;
  lucent_status st = tmp.reserve((size_t)b->node_count * 32 + (size_t)b->tri_count * 4 + 16);
  if (st) return st;
  float* ref_d = (float*)tmp.ptr;
  uint32_t* idx_d = (uint32_t*)((char*)tmp.ptr + (size_t)b->node_count * 32);
  launch_unpack((const Node*)b->nodes.ptr, b->node_count, (const float4*)b->tris.ptr, b->tri_count, ref_d, idx_d, 0);
  cudaError_t e = cudaMemcpy(nodes_out, ref_d, (size_t)b->node_count * 32, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && b->tri_count)
    e = cudaMemcpy(tri_indices_out, idx_d, (size_t)b->tri_count * 4, cudaMemcpyDeviceToHost);
  tmp.release();
  return e == cudaSuccess ? LUCENT_OK : cuda_fail(e, "download bvh");
}

lucent_status lucent_bvh_set_mode(lucent_bvh* b, int32_t mode) {
  clear_error();
  if (!b) return fail(LUCENT_ERR_INVALID, "null bvh");
  if (mode != LUCENT_TRAVERSE_FAST && mode != LUCENT_TRAVERSE_EXACT && mode != LUCENT_TRAVERSE_FAST_GLOBAL &&
      mode != LUCENT_TRAVERSE_WIDE)
    return fail(LUCENT_ERR_INVALID, "bad mode %d", mode);
  b->mode = mode;
  return LUCENT_OK;
}

lucent_status lucent_bvh_near_info(lucent_bvh* b, int32_t* usable, float* reach, uint32_t* handed_on) {
  clear_error();
  if (!b) return fail(LUCENT_ERR_INVALID, "null bvh");
  const bool near = b->views && b->near.usable;
  if (usable) *usable = near;
  if (reach) *reach = near ? b->near.bound.w : 0.f;
  if (handed_on) {
    *handed_on = 0;
    if (near && b->scratch.ptr) {  // the queue's length, the second counter word (launch_closest)
      cudaError_t e = cudaMemcpy(handed_on, (uint32_t*)b->scratch.ptr + 1, 4, cudaMemcpyDeviceToHost);
      if (e != cudaSuccess) return cuda_fail(e, "read counters");
    }
  }
  return LUCENT_OK;
}

static lucent_status check_tmin(double t_min, double t_max) {
  if (!(t_min >= 0) || std::isnan(t_max)) return fail(LUCENT_ERR_INVALID, "t_min must be >= 0 and t_max not NaN");
  return LUCENT_OK;
}

// Scratch layout: 8 counter words (launch_closest; the first is the error
// word), then 2 n words of ray queues from byte 256.
static lucent_status prepare_scratch(lucent_bvh* b, uint32_t n, cudaStream_t s, uint32_t** ctr, uint32_t** queue) {
  lucent_status st = b->scratch.reserve(256 + (size_t)n * 8);
  if (st) return st;
  *ctr = (uint32_t*)b->scratch.ptr;
  *queue = (uint32_t*)((char*)b->scratch.ptr + 256);
  cudaError_t e = cudaMemsetAsync(b->scratch.ptr, 0, 32, s);
  if (e != cudaSuccess) return cuda_fail(e, "memset scratch");
  return LUCENT_OK;
}

// The views of LUCENT_TRAVERSE_WIDE, outside any capture; returns when they
// are complete, as the next call may come on another stream.
static lucent_status build_views(lucent_bvh* b, cudaStream_t s) {
  lucent_status st;
  if (!b->near_tried) {
    if ((st = build_near_view((const Node*)b->nodes.ptr, b->node_count, (const float4*)b->tris.ptr, b->tri_count, b->lo,
                              b->hi, b->near, s)))
      return st;
    b->near_tried = true;
  }
  if (!(b->near.usable && b->near.wide_range)) {
    if ((st = b->wide.reserve((size_t)b->node_count * 4 * sizeof(Node)))) return st;
    launch_wide_view((const Node*)b->nodes.ptr, b->node_count, (Node*)b->wide.ptr, s);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e, "four-wide view");
  }
  b->views = true;
  return LUCENT_OK;
}

// Queues one call's work on s.
static lucent_status intersect_queue(lucent_bvh* b, const float* rays_d, uint32_t n, double t_min, double t_max,
                                     int32_t* prim_d, float* t_d, float* u_d, float* v_d, cudaStream_t s,
                                     bool capturing) {
  lucent_status st;
  uint32_t *ctr, *queue;
  if ((st = prepare_scratch(b, n, s, &ctr, &queue))) return st;
  if (n == 0) return LUCENT_OK;
  if (b->tri_count == 0) {  // bvh.ts:274: an empty BVH never hits
    cudaError_t e = cudaMemsetAsync(prim_d, 0xff, (size_t)n * 4, s);
    return e == cudaSuccess ? LUCENT_OK : cuda_fail(e, "memset");
  }
  if (b->mode == LUCENT_TRAVERSE_WIDE && !b->views && !capturing && (st = build_views(b, s))) return st;
  // Without them, in a capture, as mode 0: what a capture records has not run
  // by the next call, so no view can be built in one.
  const bool views = b->mode == LUCENT_TRAVERSE_WIDE && b->views;
  const bool near = views && b->near.usable;
  const Node* wide = views && !(near && b->near.wide_range) ? (const Node*)b->wide.ptr : nullptr;
  const bool top = b->mode == LUCENT_TRAVERSE_FAST || (b->mode == LUCENT_TRAVERSE_WIDE && !b->views);
  launch_closest((const Node*)b->nodes.ptr, b->node_count, (const float4*)b->tris.ptr, rays_d, n, t_min, t_max, prim_d, t_d, u_d,
                 v_d, queue, ctr, b->mode == LUCENT_TRAVERSE_EXACT || b->depth + 2 > kTsStack, top, s, wide, near ? &b->near : nullptr);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? LUCENT_OK : cuda_fail(e, "closest-hit launch");
}

lucent_status lucent_bvh_intersect_device(lucent_bvh* b, const float* rays_d, uint32_t n, double t_min,
                                          double t_max, int32_t* prim_d, float* t_d, float* u_d, float* v_d,
                                          void* stream) {
  clear_error();
  if (!b || (n && (!rays_d || !prim_d))) return fail(LUCENT_ERR_INVALID, "null argument");
  lucent_status st = check_tmin(t_min, t_max);
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaError_t e = cudaStreamIsCapturing(s, &cap); e != cudaSuccess) return cuda_fail(e, "stream");
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  if (!capturing && (st = b->uses.begin(s))) return st;
  st = intersect_queue(b, rays_d, n, t_min, t_max, prim_d, t_d, u_d, v_d, s, capturing);
  if (capturing) {  // the graph holds these from now on
    for (DeviceBuffer* m : {&b->nodes, &b->tris, &b->scratch, &b->wide, &b->near.records, &b->near.leaf_of}) m->held = true;
    return st;
  }
  const lucent_status end = b->uses.end(s);
  return st ? st : end;
}

static lucent_status device_error(unsigned word) {
  if (word & kErrIterations) return fail(LUCENT_ERR_DEVICE, "traversal exceeded node_count steps (malformed BVH)");
  if (word & kErrStack)
    return fail(LUCENT_ERR_DEVICE, "traversal needed more than 64 stack entries (BVH too deep for the reference)");
  return fail(LUCENT_ERR_DEVICE, "device error word 0x%x", word);
}

lucent_status lucent_bvh_check(lucent_bvh* b, void* stream) {
  clear_error();
  if (!b) return fail(LUCENT_ERR_INVALID, "null bvh");
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_fail(e, "synchronize");
  if (!b->scratch.ptr) return LUCENT_OK;
  unsigned word = 0;
  e = cudaMemcpy(&word, b->scratch.ptr, 4, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return cuda_fail(e, "read error word");
  if (word) {
    cudaMemset(b->scratch.ptr, 0, 4);
    return device_error(word);
  }
  return LUCENT_OK;
}

lucent_status lucent_bvh_intersect(lucent_bvh* b, const float* rays, uint32_t n, double t_min, double t_max,
                                   int32_t* prim_out, float* t_out, float* u_out, float* v_out, void* stream) {
  clear_error();
  if (!b || (n && (!rays || !prim_out))) return fail(LUCENT_ERR_INVALID, "null argument");
  if (n == 0) return LUCENT_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const size_t rb = (size_t)n * 24, ob = (size_t)n * 4;
  lucent_status st = b->stage.reserve(rb + 4 * ob + 64);
  if (st) return st;
  char* base = (char*)b->stage.ptr;
  float* rays_d = (float*)base;
  int32_t* prim_d = (int32_t*)(base + rb);
  float* t_d = (float*)(base + rb + ob);
  float* u_d = (float*)(base + rb + 2 * ob);
  float* v_d = (float*)(base + rb + 3 * ob);
  cudaError_t e = cudaMemcpyAsync(rays_d, rays, rb, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return cuda_fail(e, "upload rays");
  if ((st = lucent_bvh_intersect_device(b, rays_d, n, t_min, t_max, prim_d, t_d, u_d, v_d, stream))) return st;
  e = cudaMemcpyAsync(prim_out, prim_d, ob, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && t_out) e = cudaMemcpyAsync(t_out, t_d, ob, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && u_out) e = cudaMemcpyAsync(u_out, u_d, ob, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && v_out) e = cudaMemcpyAsync(v_out, v_d, ob, cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) {
    b->uses.unordered = true;
    return cuda_fail(e, "download hits");
  }
  if (b->tri_count == 0 && t_out)
    for (uint32_t i = 0; i < n; i++) t_out[i] = INFINITY;
  return lucent_bvh_check(b, stream);
}

lucent_status lucent_bvh_intersect_f64(lucent_bvh* b, const double* rays, uint32_t n, double t_min, double t_max,
                                       int32_t* prim_out, double* t_out, double* u_out, double* v_out,
                                       void* stream) {
  clear_error();
  if (!b || (n && (!rays || !prim_out || !t_out || !u_out || !v_out))) return fail(LUCENT_ERR_INVALID, "null argument");
  lucent_status st = check_tmin(t_min, t_max);
  if (st) return st;
  if (n == 0) return LUCENT_OK;
  if (b->tri_count == 0) {
    for (uint32_t i = 0; i < n; i++) {
      prim_out[i] = -1;
      t_out[i] = INFINITY;
      u_out[i] = v_out[i] = 0;
    }
    return LUCENT_OK;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const size_t rb = (size_t)n * 48, ob = (size_t)n * 8;
  // A warp per ray while all of them run at once (18 an SM); trees the
  // reference's stack cannot walk keep the kernel that reproduces its overflow.
  if (n <= 18 * 152 && b->depth + 2 <= kTsStack && b->mode != LUCENT_TRAVERSE_EXACT) {
    const bool args = n <= kPickArgs;
    const size_t hb = (size_t)n * sizeof(PickHit);
    if ((st = b->stage.reserve(hb + (args ? 0 : rb)))) return st;
    PickHit* hits_d = (PickHit*)b->stage.ptr;
    double* rays_d = (double*)((char*)b->stage.ptr + hb);
    cudaError_t e = args ? cudaSuccess : cudaMemcpyAsync(rays_d, rays, rb, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_fail(e, "upload rays");
    launch_pick((const Node*)b->nodes.ptr, b->node_count, (const float4*)b->tris.ptr, args ? rays : rays_d, !args, n,
                t_min, t_max, hits_d, s);
    PickHit few[kPickArgs];
    std::vector<PickHit> many(args ? 0 : n);
    PickHit* hits = args ? few : many.data();
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hits, hits_d, hb, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      b->uses.unordered = true;
      return cuda_fail(e, "f64 closest-hit");
    }
    unsigned word = 0;
    for (uint32_t i = 0; i < n; i++) {
      prim_out[i] = hits[i].prim;
      t_out[i] = hits[i].t;
      u_out[i] = hits[i].u;
      v_out[i] = hits[i].v;
      word |= hits[i].err;
    }
    return word ? device_error(word) : LUCENT_OK;
  }
  if ((st = b->stage.reserve(rb + 4 * ob + 64))) return st;
  uint32_t *ctr, *queue;
  if ((st = prepare_scratch(b, 0, s, &ctr, &queue))) return st;
  char* base = (char*)b->stage.ptr;
  double* rays_d = (double*)base;
  int32_t* prim_d = (int32_t*)(base + rb);
  double* t_d = (double*)(base + rb + ob);
  double* u_d = (double*)(base + rb + 2 * ob);
  double* v_d = (double*)(base + rb + 3 * ob);
  cudaError_t e = cudaMemcpyAsync(rays_d, rays, rb, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return cuda_fail(e, "upload rays");
  launch_closest_d((const Node*)b->nodes.ptr, b->node_count, (const float4*)b->tris.ptr, rays_d, n, t_min, t_max, prim_d, t_d, u_d,
                   v_d, ctr, s);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(prim_out, prim_d, (size_t)n * 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(t_out, t_d, ob, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(u_out, u_d, ob, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(v_out, v_d, ob, cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) {
    b->uses.unordered = true;
    return cuda_fail(e, "f64 closest-hit");
  }
  return lucent_bvh_check(b, stream);
}

}  // extern "C"
