// softplus of the KDA log-decay gate, shared by the element-wise kernel and the projection that ends in it.
#pragma once
#include "common.cuh"

namespace daisy {

__device__ __forceinline__ float round_bf16(float x) { return __uint_as_float(pack_bf16(0.f, x) & 0xffff0000u); }
// log1p(u), u in [0, 1]: degree-9 polynomial for log1p(u) / u (Chebyshev interpolant; 1.6e-7 relative in fp32 arithmetic)
__device__ constexpr float LOG1P_C[10] = {-0.0031760570127516985f, 0.019542528316378593f, -0.05637361481785774f, 0.10543623566627502f, -0.1526966691017151f,
                                          0.1966327428817749f, -0.24951615929603577f, 0.33329710364341736f, -0.49999892711639404f, 1.0f};
__device__ __forceinline__ float log1p_unit(float u) {
  float r = LOG1P_C[0];
#pragma unroll
  for (int k = 1; k < 10; ++k) r = fmaf(r, u, LOG1P_C[k]);
  return r * u;
}
// softplus(beta x) / beta as  max(z, 0) + log1p(u),  u = exp(-|z|) in (0, 1]  with one ex2.approx; x itself above the threshold
__device__ __forceinline__ float kda_softplus(float x, float beta, float inv_beta, float threshold) {
  const float z = x * beta, u = fast_exp2(fabsf(z) * -1.4426950408889634f);
  return z > threshold ? x : (fmaxf(z, 0.f) + log1p_unit(u)) * inv_beta;
}

}  // namespace daisy
