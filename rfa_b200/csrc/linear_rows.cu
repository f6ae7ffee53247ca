// Projections of a few rows:  y_m = x W_m^T + b_m  for one to three matrices of one shape, fp16 in and out, fp32 sums -- the
// q / k / v and output projections of a layer that decodes one token for a batch (nn.Linear in upstream,
// causal_attention.py:222-239, 277-280).
//
// Bound by the weights' way from L2 or HBM (3 x 1024 x 1024: 6 MB, 1 us at 6.5 TB/s) and, in a program, by launches: four cuBLAS calls,
// two for sigma * W and seven launches in all were 108 us a token and layer at batch 8 x 16 heads, nearly all of it host
// time.  One launch here takes all matrices that share x, and forms the step's effective random matrices on the way in blocks of its own:
// three launches a token, 12.7 us of kernels (two of these 6.1, the decoding step 6.6) instead of 30, and 24.5 us a pass instead of 102.
//
// A row of y is short work, so the sum over the inner index is split over the warps of a CTA: a warp takes 32 of it at a time for
// 16 MT rows of W against 8 NT tokens.  mma.sync m16n8k16 with the W rows as A; the order of the inner index is free, so lane t of a
// quad stands for elements 8t .. 8t + 7 of the 32 and a fragment is one 16-byte load of W (64 contiguous bytes a row) and one of
// x, straight from global memory: W is read once by one warp, x stays in L1 / L2.  All loads of four (two) steps are issued before the
// first product.  tcgen05 would stage both through shared memory for M = 128 rows of which a batch of 8 fills 8.
// The warps' sums meet in shared memory in fp32, so that a chain inside the mma's truncating accumulators is 1/8 (1/4) of
// the inner index.
#include "matrices.cuh"
#include "sm100.cuh"

namespace rfa {

constexpr int kLrThreads = 256, kLrMax = 3;
struct LrArgs {
  const __half *w[kLrMax], *b[kLrMax];
  __half* y[kLrMax];
};

__device__ __forceinline__ void lr_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// grid (matrix blocks + count * row tiles, token groups).  KS: parts the inner index is split into; the other 8 / KS warps take
// further tokens.  U: steps of 32 in flight.
template <int MT, int NT, int KS, int U>
__global__ void __launch_bounds__(kLrThreads, 2)
linear_rows_kernel(const __half* __restrict__ x, const __grid_constant__ LrArgs a, int tiles, int n, int in, int out,
                   const __grid_constant__ LrMatrices m, int m_blocks) {
  constexpr int kRows = 16 * MT, kTok = 8 * NT * (8 / KS);
  __shared__ float red[KS][kTok][kRows + 4];
  sm100::pdl_wait();
  sm100::pdl_launch_dependents();
  if (blockIdx.x < (unsigned)m_blocks) {
    if (blockIdx.y == 0) lr_matrices<kLrThreads>(m, blockIdx.x, m_blocks);
    return;
  }
  const int tile = blockIdx.x - m_blocks, which = tile / tiles, row0 = (tile % tiles) * kRows, tok0 = blockIdx.y * kTok;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ks = warp % KS, my_tok = tok0 + (warp / KS) * 8 * NT;
  const __half* w = a.w[which];
  const uint4 zero = make_uint4(0, 0, 0, 0);
  float acc[MT][NT][4] = {};
  for (int k0 = ks * 32; k0 < in; k0 += KS * 32 * U) {
    uint4 fa[U][MT][2], fb[U][NT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + u * KS * 32 + 8 * t;
      const bool live = k < in;
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int row = row0 + 16 * i + 8 * r + g;
          fa[u][i][r] = live && row < out ? *reinterpret_cast<const uint4*>(w + (size_t)row * in + k) : zero;
        }
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int tok = my_tok + 8 * j + g;
        fb[u][j] = live && tok < n ? *reinterpret_cast<const uint4*>(x + (size_t)tok * in + k) : zero;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const uint4 p = fa[u][i][0], q = fa[u][i][1], b = fb[u][j];
          lr_mma(acc[i][j], p.x, q.x, p.y, q.y, b.x, b.y);
          lr_mma(acc[i][j], p.z, q.z, p.w, q.w, b.z, b.w);
        }
  }
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)      // accumulator e: W row g (+ 8), token 2t (+ 1)
        red[ks][(warp / KS) * 8 * NT + 8 * j + 2 * t + (e & 1)][16 * i + g + 8 * (e >> 1)] = acc[i][j][e];
  __syncthreads();
  for (int i = threadIdx.x; i < kTok * kRows / 2; i += kLrThreads) {
    const int tok = i / (kRows / 2), r = (i % (kRows / 2)) * 2;
    if (tok0 + tok >= n || row0 + r >= out) continue;          // out is even
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 0; k < KS; ++k) { s.x += red[k][tok][r]; s.y += red[k][tok][r + 1]; }
    if (a.b[which]) {
      const float2 b = __half22float2(*reinterpret_cast<const __half2*>(a.b[which] + row0 + r));
      s.x += b.x; s.y += b.y;
    }
    *reinterpret_cast<__half2*>(a.y[which] + (size_t)(tok0 + tok) * out + row0 + r) = __floats2half2_rn(s.x, s.y);
  }
}

template <int MT, int NT, int KS, int U>
static int lr_launch(const __half* x, const LrArgs& a, int count, int n, int in, int out, const LrMatrices& m, cudaStream_t st) {
  const int tiles = (out + 16 * MT - 1) / (16 * MT), tok = 8 * NT * (8 / KS), m_blocks = (m.n + kLrThreads * 8 - 1) / (kLrThreads * 8);
  sm100::launch_pdl(linear_rows_kernel<MT, NT, KS, U>, dim3(count * tiles + m_blocks, (n + tok - 1) / tok), dim3(kLrThreads), 0, st, x, a, tiles,
                    n, in, out, m, m_blocks);
  return check_launch("rfa_linear_rows");
}

}  // namespace rfa

using namespace rfa;

extern "C" int rfa_linear_rows(const void* x, const void* const* w, const void* const* b, void* const* y, int count, int n, int in, int out,
                               const void* rm, const void* sigma, float inv_tau, float* w_eff, int H, int D, int d, rfa_stream_t stream) {
  RFA_REQUIRE(count >= 1 && count <= kLrMax && n >= 0 && in > 0 && out > 0, RFA_EINVAL, "linear_rows: count=%d n=%d in=%d out=%d", count, n, in, out);
  RFA_REQUIRE(in % 8 == 0 && out % 8 == 0 && n <= 65535, RFA_EUNSUPPORTED, "linear_rows: in=%d and out=%d must be multiples of 8, n=%d at most 65535",
              in, out, n);
  RFA_REQUIRE(w && b && y && (n == 0 || x), RFA_EINVAL, "linear_rows: null pointer");
  LrArgs a{};
  for (int i = 0; i < count; ++i) {
    RFA_REQUIRE(w[i] && (n == 0 || y[i]), RFA_EINVAL, "linear_rows: null pointer");
    RFA_REQUIRE(aligned16(w[i]) && aligned16(b[i]) && aligned16(y[i]), RFA_EALIGN, "linear_rows: 16-byte alignment required");
    a.w[i] = (const __half*)w[i]; a.b[i] = (const __half*)b[i]; a.y[i] = (__half*)y[i];
  }
  LrMatrices m{};
  if (rm) {
    RFA_REQUIRE(w_eff && H > 0 && D > 0 && d > 0, RFA_EINVAL, "linear_rows: matrices want w_eff and H=%d, D=%d, d=%d positive", H, D, d);
    RFA_REQUIRE(d % 8 == 0 && (int64_t)H * D * d < (1 << 30), RFA_EUNSUPPORTED, "linear_rows: matrices H=%d D=%d d=%d", H, D, d);
    m = LrMatrices{(const __half*)rm, (const __half*)sigma, w_eff, inv_tau, H * D * d, D * d, d};
  }
  RFA_REQUIRE(aligned16(x) && aligned16(rm) && aligned16(sigma) && aligned16(w_eff), RFA_EALIGN, "linear_rows: 16-byte alignment required");
  if (n == 0) return 0;
  cudaStream_t st = as_stream(stream);
  const __half* xh = (const __half*)x;
  // Rows of W a CTA holds against tokens: W is read once per token group and x once per row tile, both from L2.  Up to 32 tokens
  // one group of narrow tiles (more CTAs); beyond, 32 rows x 64 tokens halve the traffic of x.
  if (n <= 8) return lr_launch<1, 1, 8, 4>(xh, a, count, n, in, out, m, st);
  if (n <= 16) return lr_launch<1, 2, 8, 4>(xh, a, count, n, in, out, m, st);
  if (n <= 32) return lr_launch<1, 4, 8, 2>(xh, a, count, n, in, out, m, st);
  return lr_launch<2, 4, 4, 2>(xh, a, count, n, in, out, m, st);
}
