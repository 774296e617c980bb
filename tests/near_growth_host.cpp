// leaf_growth of the nearest-first view, as the host compiles it.
#include "near_growth.h"

extern "C" void growth(const float* tri, int n, float s, float* out, float* rise) {
  for (int k = 0; k < n; k++) {
    const float* v = tri + 9 * k;
    rise[k] = 0.f;
    out[k] = lucent::leaf_growth({v[0], v[1], v[2], 0.f}, {v[3], v[4], v[5], 0.f}, {v[6], v[7], v[8], 0.f}, s, rise[k]);
  }
}
