// Host-side helpers shared by the C ABI translation units.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/lucent.h"

namespace lucent {

lucent_status fail(lucent_status code, const char* fmt, ...);
lucent_status cuda_fail(cudaError_t e, const char* what);
void clear_error();

// Index of the first infinity or NaN in v[0 .. n - 1], or n.
uint64_t first_not_finite(const float* v, uint64_t n);

// A growable device allocation owned by a handle.
struct DeviceBuffer {
  void* ptr = nullptr;
  size_t cap = 0;
  bool pooled = false;  // from the pool (TempBuffer) instead of cudaMalloc
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

}  // namespace lucent

extern "C" {
// Reference-layout BVH checks shared by the C-ABI files (defined in api.cu).
uint32_t tree_depth(const float* nodes, uint32_t node_count, uint32_t tri_count);
lucent_status validate_bvh(const float* nodes, uint32_t node_count, const uint32_t* tri, uint32_t tri_count);
}
