// The effective random matrices of a layer:  w_eff[h][j][l] = round(sigma[h][l] * rm[h][j][l]) (sigma null: rm) * inv_tau, rounded again
// where inv_tau is not 1 -- the fp16 roundings of the tensor expressions they replace (build_random_matrices, utils.py:90-97).
#pragma once

#include "common.cuh"

namespace rfa {

struct LrMatrices {
  const __half *rm, *sigma;
  float* w_eff;
  float inv_tau;
  int n, Dd, d;      // elements in all, per head, per row
};

template <int THREADS>
__device__ __forceinline__ void lr_matrices(const LrMatrices& m, int block, int blocks) {
  for (int i = (block * THREADS + threadIdx.x) * 8; i < m.n; i += blocks * THREADS * 8) {      // 8 | d: a piece is of one row
    float w[8];
    load8(m.rm + i, w);
    if (m.sigma) {
      float s[8];
      load8(m.sigma + (size_t)(i / m.Dd) * m.d + i % m.d, s);
#pragma unroll
      for (int e = 0; e < 8; ++e) w[e] = __half2float(__float2half_rn(w[e] * s[e]));
    }
    if (m.inv_tau != 1.f)
#pragma unroll
      for (int e = 0; e < 8; ++e) w[e] = __half2float(__float2half_rn(w[e] * m.inv_tau));
    store4(m.w_eff + i, make_float4(w[0], w[1], w[2], w[3]));
    store4(m.w_eff + i + 4, make_float4(w[4], w[5], w[6], w[7]));
  }
}

}  // namespace rfa
