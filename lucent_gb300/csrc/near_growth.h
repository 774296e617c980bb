// By how much the nearest-first view grows a triangle's leaf box. Plain
// arithmetic for the host and the device.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace lucent {

// How far outside triangle (a, b, c) the reference's binary64 test may accept
// a point o + t d (the derivation is at the top of traverse_near.cuh), for
// |d| <= 2 and |o - v0| <= s, and by how much that rises per unit of s. kHuge:
// edges so long that |det| >= 1e-12 bounds nothing.
//
// In binary32, rounded up: edges are off by 2^-24 of themselves, so lengths by
// far less than 1e-5 (and 1e-18 where squares leave the normal range), and the
// cross product by less than 1e-6 |e1| |e2| (three roundings of terms at most
// that large, in three components). Where that leaves open whether a triangle
// in a coordinate plane is thin, it gets the growth of one that is. In binary64
// k_near_leaves over 2,000,000 triangles took 355 us, so 131.
constexpr float kHuge = 1e30f;
__host__ __device__ inline float leaf_growth(float4 a, float4 b, float4 c, float s, float& rise) {
  const float e1x = b.x - a.x, e1y = b.y - a.y, e1z = b.z - a.z;
  const float e2x = c.x - a.x, e2y = c.y - a.y, e2z = c.z - a.z;
  const float nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
  const float l1 = sqrtf(e1x * e1x + e1y * e1y + e1z * e1z) * 1.00001f + 1e-18f;
  const float l2 = sqrtf(e2x * e2x + e2y * e2y + e2z * e2z) * 1.00001f + 1e-18f;
  const float reach = 4.f * s + 3.f * fmaxf(l1, l2);  // 3 |s| + t |d| + |e1| + |e2|
  const float ll = l1 * l2, nn = nx * nx + ny * ny + nz * nz;
  const bool flat = (a.x == b.x && a.x == c.x) || (a.y == b.y && a.y == c.y) || (a.z == b.z && a.z == c.z);
  float k = 3.7252903e-09f;  // 2^-28
  if (!(flat && nn > 1e-30f && ll < 65000.f * (sqrtf(nn) - 1e-6f * ll))) {
    const float w = 2.1e-3f * ll / fmaxf(1.f - 1.8e-3f * ll, 1e-6f);
    if (!(w < 0.5f)) return kHuge;
    k += w / (1.f - w);
  }
  rise = fmaxf(rise, 4.f * k);
  return k * reach;
}

}  // namespace lucent
