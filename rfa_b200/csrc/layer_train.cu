// What a layer's training step needs besides its products, features and attention: the gradients of the projections' biases, the
// step's random matrices from sigma and their gradient.  (nn.Linear's and build_random_matrices' backward in upstream,
// causal_attention.py:222-239, utils.py:90-97.)
//
// All of it is small and was bound by launches: one reduction per bias (9 us each for 3600 x 512, of which 0.6 us are the bytes), and for
// sigma * W a product, two conversions, a sum and two more products.  Here one launch makes the sums of up to three
// gradients, one the matrices and the transposed padding mask, one both gradients of the matrices.
// A training step of 24 x 150 tokens in 8 heads: 35 launches -> 22, kernels 223 -> 165 us (column sums 45.8 -> 8.8), 698 -> 465 us a
// step; 8 x 2048 tokens in 16 heads 858 -> 757.
#include <cooperative_groups.h>

#include "matrices.cuh"

namespace rfa {
namespace cg = cooperative_groups;

// ---- out_m[c] = sum over rows of g_m[row][c] ---------------------------------------------------------------------------------
// Bound by memory.  A cluster of eight CTAs takes 32 columns (64 bytes of a row, two sectors) and an eighth of the rows each: a layer of
// 512 features is 128 CTAs a gradient, each with 32 KB on the way.  fp32 throughout, in a fixed order: 512 chains of a
// thread, then warp, CTA and cluster.
constexpr int kCsThreads = 256, kCsMax = 3, kCsCluster = 8, kCsCols = 32, kCsRows = kCsThreads / (kCsCols / 8), kCsFlight = 8;
struct CsArgs {
  const __half* g[kCsMax];
  __half* out[kCsMax];
};
__global__ void __cluster_dims__(kCsCluster, 1, 1) __launch_bounds__(kCsThreads)
column_sums_kernel(const __grid_constant__ CsArgs a, int64_t rows, int cols) {
  __shared__ float red[kCsThreads / 32][kCsCols], part[kCsCols];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = blockIdx.x % kCsCluster, col0 = blockIdx.x / kCsCluster * kCsCols, c = col0 + (threadIdx.x & 3) * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const __half* g = a.g[blockIdx.y];
  float acc[8] = {};
  if (c < cols) {                                      // 8 | cols
    const int64_t end = rows * (rank + 1) / kCsCluster;
    for (int64_t r = rows * rank / kCsCluster + (threadIdx.x >> 2); r < end; r += kCsRows * kCsFlight) {
      uint4 u[kCsFlight];
#pragma unroll
      for (int i = 0; i < kCsFlight; ++i)
        u[i] = r + i * kCsRows < end ? __ldg(reinterpret_cast<const uint4*>(g + (size_t)(r + i * kCsRows) * cols + c)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int i = 0; i < kCsFlight; ++i) {
        const uint32_t w[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
          acc[2 * e] += f.x; acc[2 * e + 1] += f.y;
        }
      }
    }
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
  if (lane < 4)
#pragma unroll
    for (int e = 0; e < 8; ++e) red[warp][lane * 8 + e] = acc[e];
  __syncthreads();
  if (threadIdx.x < kCsCols) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kCsThreads / 32; ++w) s += red[w][threadIdx.x];
    part[threadIdx.x] = s;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x < kCsCols && col0 + threadIdx.x < cols) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < kCsCluster; ++r) s += *cluster.map_shared_rank(part + threadIdx.x, r);
    a.out[blockIdx.y][col0 + threadIdx.x] = __float2half_rn(s);
  }
  cluster.sync();                                      // the others' shared memory stays until it has been read
}

// ---- the matrices and the padding mask as the feature map takes it: row_mask[t][b] = pad[b][t] ------------------------------------
constexpr int kLmThreads = 256;
__global__ void __launch_bounds__(kLmThreads)
layer_matrices_kernel(const __grid_constant__ LrMatrices m, int m_blocks, const uint8_t* __restrict__ pad, uint8_t* __restrict__ row_mask, int64_t T,
                      int B) {
  if ((int)blockIdx.x < m_blocks) {
    lr_matrices<kLmThreads>(m, blockIdx.x, m_blocks);
    return;
  }
  const int64_t i = (int64_t)(blockIdx.x - m_blocks) * kLmThreads + threadIdx.x;
  if (i < T * B) row_mask[i] = pad[i % B * T + i / B];
}

// ---- g_sigma[h][l] = sum_j g[h][j][l] rm[h][j][l] inv_tau,  g_rm = g sigma inv_tau; a CTA a head, 8 columns a thread ------------------
__global__ void __launch_bounds__(kLmThreads)
layer_matrices_bwd_kernel(const float* __restrict__ g, const __half* __restrict__ rm, const __half* __restrict__ sigma, float inv_tau,
                          __half* __restrict__ g_sigma, __half* __restrict__ g_rm, int D, int d) {
  __shared__ float red[kLmThreads * 8];                // [rows in flight][d]
  const int h = blockIdx.x, pieces = d / 8, lines = kLmThreads / pieces, l = threadIdx.x % pieces * 8, line = threadIdx.x / pieces;
  const size_t base = (size_t)h * D * d;
  float s[8], acc[8] = {};
#pragma unroll
  for (int e = 0; e < 8; ++e) s[e] = 1.f;
  if (sigma) load8(sigma + (size_t)h * d + l, s);
  if (line < lines) {
    for (int j = line; j < D; j += lines) {
      const size_t at = base + (size_t)j * d + l;
      const float4 x = load4(g + at), y = load4(g + at + 4);
      const float v[8] = {x.x * inv_tau, x.y * inv_tau, x.z * inv_tau, x.w * inv_tau, y.x * inv_tau, y.y * inv_tau, y.z * inv_tau, y.w * inv_tau};
      if (g_sigma) {
        float w[8];
        load8(rm + at, w);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] = fmaf(v[e], w[e], acc[e]);
      }
      if (g_rm) {
        store4(g_rm + at, make_float4(v[0] * s[0], v[1] * s[1], v[2] * s[2], v[3] * s[3]));
        store4(g_rm + at + 4, make_float4(v[4] * s[4], v[5] * s[5], v[6] * s[6], v[7] * s[7]));
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) red[line * d + l + e] = acc[e];
  }
  __syncthreads();
  if (g_sigma && (int)threadIdx.x < d) {
    float sum = 0.f;
    for (int i = 0; i < lines; ++i) sum += red[i * d + threadIdx.x];
    g_sigma[(size_t)h * d + threadIdx.x] = __float2half_rn(sum);
  }
}

}  // namespace rfa

using namespace rfa;

extern "C" int rfa_column_sums(const void* const* g, void* const* out, int count, int64_t rows, int cols, rfa_stream_t stream) {
  RFA_REQUIRE(g && out, RFA_EINVAL, "column_sums: null pointer");
  RFA_REQUIRE(count > 0 && count <= kCsMax && rows >= 0 && cols > 0, RFA_EINVAL, "column_sums: count=%d rows=%lld cols=%d", count, (long long)rows, cols);
  RFA_REQUIRE(cols % 8 == 0, RFA_EUNSUPPORTED, "column_sums: need cols%%8==0 (got %d)", cols);
  CsArgs a{};
  for (int m = 0; m < count; ++m) {
    RFA_REQUIRE(out[m] && (g[m] || rows == 0), RFA_EINVAL, "column_sums: null pointer");
    RFA_REQUIRE(aligned16(g[m]), RFA_EALIGN, "column_sums: 16-byte alignment required");
    a.g[m] = (const __half*)g[m];
    a.out[m] = (__half*)out[m];
  }
  column_sums_kernel<<<dim3((unsigned)((cols + kCsCols - 1) / kCsCols) * kCsCluster, count), kCsThreads, 0, as_stream(stream)>>>(a, rows, cols);
  return check_launch("rfa_column_sums");
}

extern "C" int rfa_layer_matrices(const void* rm, const void* sigma, float inv_tau, float* w_eff, int H, int D, int d, const uint8_t* pad_mask,
                                  uint8_t* row_mask, int64_t T, int B, rfa_stream_t stream) {
  RFA_REQUIRE(rm && w_eff && (!pad_mask || row_mask), RFA_EINVAL, "layer_matrices: null pointer");
  RFA_REQUIRE(H > 0 && D > 0 && d > 0 && T >= 0 && B >= 0, RFA_EINVAL, "layer_matrices: H=%d D=%d d=%d T=%lld B=%d", H, D, d, (long long)T, B);
  RFA_REQUIRE(d % 8 == 0 && (int64_t)H * D * d <= (1 << 30), RFA_EUNSUPPORTED, "layer_matrices: need d%%8==0 (got %d), at most 2^30 elements", d);
  RFA_REQUIRE(aligned16(rm) && aligned16(sigma) && aligned16(w_eff), RFA_EALIGN, "layer_matrices: 16-byte alignment required");
  const int n = H * D * d;
  const int64_t mask_blocks = pad_mask ? (T * B + kLmThreads - 1) / kLmThreads : 0;
  RFA_REQUIRE(mask_blocks < (1 << 30), RFA_EUNSUPPORTED, "layer_matrices: T * B = %lld", (long long)(T * B));
  const int want = (n / 8 + kLmThreads - 1) / kLmThreads, m_blocks = want < 592 ? want : 592;
  layer_matrices_kernel<<<(unsigned)(m_blocks + mask_blocks), kLmThreads, 0, as_stream(stream)>>>(
      LrMatrices{(const __half*)rm, (const __half*)sigma, w_eff, inv_tau, n, D * d, d}, m_blocks, pad_mask, row_mask, T, B);
  return check_launch("rfa_layer_matrices");
}

extern "C" int rfa_layer_matrices_bwd(const float* g_w, const void* rm, const void* sigma, float inv_tau, void* g_sigma, void* g_rm, int H, int D, int d,
                                      rfa_stream_t stream) {
  RFA_REQUIRE(g_w && (!g_sigma || rm), RFA_EINVAL, "layer_matrices_bwd: null pointer");
  RFA_REQUIRE(H > 0 && D > 0 && d > 0, RFA_EINVAL, "layer_matrices_bwd: H=%d D=%d d=%d", H, D, d);
  RFA_REQUIRE(d % 8 == 0 && d <= kLmThreads, RFA_EUNSUPPORTED, "layer_matrices_bwd: need d%%8==0, d<=%d (got %d)", kLmThreads, d);
  RFA_REQUIRE(aligned16(g_w) && aligned16(rm) && aligned16(sigma) && aligned16(g_rm), RFA_EALIGN, "layer_matrices_bwd: 16-byte alignment required");
  if (!g_sigma && !g_rm) return 0;
  layer_matrices_bwd_kernel<<<(unsigned)H, kLmThreads, 0, as_stream(stream)>>>(g_w, (const __half*)rm, (const __half*)sigma, inv_tau, (__half*)g_sigma,
                                                                             (__half*)g_rm, D, d);
  return check_launch("rfa_layer_matrices_bwd");
}
