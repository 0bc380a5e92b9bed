// Top-2 routing of one token by one warp, shared by the router kernels.
#pragma once
#include <cuda_runtime.h>

#include "rbv/moe.h"

namespace rbv {

struct Top2 { int e[2]; float w[2]; };   // the same on every lane

// Softmax over E logits, the two largest (lower index wins ties), weights renormalised to sum to one.
__device__ __forceinline__ Top2 route_token(const float* __restrict__ row, int E, int lane) {
  float v[kMoeMaxExperts / 32];
  float mx = -INFINITY;
  #pragma unroll
  for (int j = 0; j < kMoeMaxExperts / 32; j++) {
    int e = j * 32 + lane;
    v[j] = e < E ? row[e] : -INFINITY;
    mx = fmaxf(mx, v[j]);
  }
  #pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  // top-2 by (value, lower index wins ties)
  float best[2]; int bi[2];
  #pragma unroll
  for (int k = 0; k < 2; k++) {
    float bv = -INFINITY; int be = 0x7fffffff;
    #pragma unroll
    for (int j = 0; j < kMoeMaxExperts / 32; j++) {
      int e = j * 32 + lane;
      bool taken = (k == 1 && e == bi[0]);
      if (e < E && !taken && (v[j] > bv || (v[j] == bv && e < be))) { bv = v[j]; be = e; }
    }
    #pragma unroll
    for (int o = 16; o; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ov > bv || (ov == bv && oe < be)) { bv = ov; be = oe; }
    }
    if (be >= E) be = (k == 1 && bi[0] == 0) ? 1 : 0;   // a row of NaN has no largest value: any expert, but a valid one
    best[k] = bv; bi[k] = be;
  }
  // softmax probabilities of the two winners, renormalised: p_k / (p_0 + p_1)
  const float p0 = __expf(best[0] - mx), p1 = __expf(best[1] - mx);
  const float inv = 1.0f / (p0 + p1);
  return Top2{{bi[0], bi[1]}, {p0 * inv, p1 * inv}};
}

}  // namespace rbv
