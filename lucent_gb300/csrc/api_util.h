// Host-side helpers shared by the C ABI translation units.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <shared_mutex>
#include <vector>

#include "../../include/lucent.h"

namespace lucent {

lucent_status fail(lucent_status code, const char* fmt, ...);
lucent_status cuda_fail(cudaError_t e, const char* what);
void clear_error();

// Index of the first infinity or NaN in v[0 .. n - 1], or n.
uint64_t first_not_finite(const float* v, uint64_t n);

struct Pool;  // a device's memory pool (api.cu)

// The work that may still use a handle's pooled memory: the last call queued on
// each stream, as events. Memory given back is ordered behind them on the
// pool's stream, so nothing waits on the host, whatever device or thread
// gives it back, and another thread's capture is not disturbed.
struct StreamUses {
  struct Use {
    unsigned long long stream;
    cudaEvent_t event;
    bool open;  // recorded, and not yet waited for by the pool's stream
  };
  Pool* home = nullptr;      // where the memory comes from, from the first reserve on
  std::vector<Use> uses;     // a few streams; the oldest makes room
  std::vector<void*> kept;   // given back while a graph may hold them, until close()
  bool unordered = false;    // a call failed midway: its work has no event
  lucent_status begin(cudaStream_t s);  // before a call queues work on s, outside a capture
  lucent_status end(cudaStream_t s);    // behind that work
  void give_back(void* ptr, bool held);
  void close();  // with the handle
};

// A growable device allocation owned by a handle: from the pool where `uses`
// is given, else from cudaMalloc.
struct DeviceBuffer {
  void* ptr = nullptr;
  size_t cap = 0;
  StreamUses* uses = nullptr;
  bool held = false;  // pooled: a captured graph holds the address
  lucent_status reserve(size_t bytes);
  void release();
};

// Device memory of one call, from a stream-ordered pool that keeps what is
// freed for the next: released on the stream it was reserved on.
struct TempBuffer {
  void* ptr = nullptr;
  cudaStream_t stream = nullptr;
  lucent_status reserve(size_t bytes, cudaStream_t s);
  void release();
};
void trim_temporaries();  // gives the pool's free memory back

// Held shared while this library captures a graph: a device cannot be
// synchronised then.
std::shared_mutex& capture_lock();

}  // namespace lucent

extern "C" {
// Reference-layout BVH checks shared by the C-ABI files (defined in api.cu).
uint32_t tree_depth(const float* nodes, uint32_t node_count, uint32_t tri_count);
lucent_status validate_bvh(const float* nodes, uint32_t node_count, const uint32_t* tri, uint32_t tri_count);
}
