// Fused random feature map and its gradient on register tiles: widths above 64, and few rows (the rest: feature_map_mma.cu,
// feature_map_tc.cu).
//
//   n = |x|_2,  xh = x / (n + 1e-3),  u = W_h xh,  phi = scale * [sin u | cos u]
// (upstream utils.py:100-120, one pass instead of norm/div/einsum/sin/cos/cat/mul).
// x [rows,H,d], W [H,D,d] fp32, phi [rows,H,2D].  One CTA owns one head and walks
// tiles of 64 rows with that head's W resident in shared memory; each x element is
// read once and each phi element written once.
#include "common.cuh"
#include "trig.cuh"

namespace rfa {

constexpr int kFmThreads = 256;
// Bound by fp32 arithmetic at 64 x 64 (3 of 4 products' FMAs are in the backward) and by memory at 32 x 32.  The products are
// register tiles of 4 x 4 fed by 16-byte shared-memory reads (8 reads, 12 wavefronts, per 64 FMAs and warp; one 4-byte
// read per operand element kept the load/store unit busy twice as long as the FMA pipe), and what follows a product
// happens in its registers: the sines and cosines of u go straight to phi, g_u straight to the operand of the next two
// products, and x_hat . g_xh is taken as sum_j g_u[j] u[j], which is at hand, not as a pass over g_xh.
//
// A thread owns rows rg + 16 i (rg = tid / 16) and columns 4 (tid % 16) .. + 3 of each block of 64 columns.  Pitches are
// the width + 4: rows one apart are 4 banks apart and stay 16-byte aligned.
//
// NI rows a thread, 16 NI a tile: 64 of them, or 32 in a backward whose tiles of 64 would leave SMs idle (see its launch).

struct FmSmem {
  float* Wt;   // [d][D + 4]   W transposed
  float* X;    // [rows][d + 4]  normalised rows
  float* nrm;  // [rows]
  float* W;    // [D][d + 4]   (backward)
  float* GU;   // [rows][D + 4]  (backward)
  float* c2;   // [rows]         (backward) x_hat . g_xh
};
__host__ __device__ inline size_t fm_smem_floats(int rows, int D, int d, bool bwd) {
  const size_t fwd = (size_t)d * (D + 4) + (size_t)rows * (d + 4) + rows;
  return bwd ? fwd + (size_t)D * (d + 4) + (size_t)rows * (D + 4) + rows : fwd;
}
__device__ __forceinline__ FmSmem fm_carve(float* base, int rows, int D, int d) {
  FmSmem s;
  s.Wt = base;
  s.X = s.Wt + d * (D + 4);
  s.nrm = s.X + rows * (d + 4);
  s.W = s.nrm + rows;
  s.GU = s.W + D * (d + 4);
  s.c2 = s.GU + rows * (D + 4);
  return s;
}

// Load + normalise a tile of rows of this head into s.X (zero rows past the end): 16 lanes per row, all of a thread's loads issued
// before the first sum.
template <int NI, typename TX>
__device__ __forceinline__ void fm_load_rows(const FmSmem& s, const TX* __restrict__ x, int64_t row0, int64_t rows, int H, int h, int d) {
  const int rg = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  float4 v[NI][2];
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t row = row0 + rg + 16 * i;
      v[i][u] = row < rows && c + 64 * u < d ? load4(x + ((size_t)row * H + h) * d + c + 64 * u) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    float ss = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) ss = fmaf(v[i][u].x, v[i][u].x, fmaf(v[i][u].y, v[i][u].y, fmaf(v[i][u].z, v[i][u].z, fmaf(v[i][u].w, v[i][u].w, ss))));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float n = sqrtf(ss), inv = 1.f / (n + kNormEps);
    const int r = rg + 16 * i;
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (c + 64 * u < d)
        store4(s.X + r * (d + 4) + c + 64 * u, make_float4(v[i][u].x * inv, v[i][u].y * inv, v[i][u].z * inv, v[i][u].w * inv));
    if (c == 0) s.nrm[r] = n;
  }
}
__device__ __forceinline__ void fm_axpy(float (&acc)[4], float a, float4 b) {
  acc[0] = fmaf(a, b.x, acc[0]); acc[1] = fmaf(a, b.y, acc[1]); acc[2] = fmaf(a, b.z, acc[2]); acc[3] = fmaf(a, b.w, acc[3]);
}
// acc[i][.] = sum_l A[rg + 16 i][l] B[l][col .. col + 3]
template <int NI>
__device__ __forceinline__ void fm_product(float (&acc)[NI][4], const float* A, int pa, const float* B, int pb, int L, int rg, int col) {
#pragma unroll
  for (int i = 0; i < NI; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
#pragma unroll 2
  for (int l = 0; l < L; l += 4) {
    float4 a[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) a[i] = load4(A + (rg + 16 * i) * pa + l);
    const float4 b0 = load4(B + l * pb + col), b1 = load4(B + (l + 1) * pb + col), b2 = load4(B + (l + 2) * pb + col), b3 = load4(B + (l + 3) * pb + col);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      fm_axpy(acc[i], a[i].x, b0); fm_axpy(acc[i], a[i].y, b1); fm_axpy(acc[i], a[i].z, b2); fm_axpy(acc[i], a[i].w, b3);
    }
  }
}

template <typename TX, typename TP>
__global__ void __launch_bounds__(kFmThreads, 4)
feature_map_fwd_kernel(const TX* __restrict__ x, const float* __restrict__ w, const uint8_t* __restrict__ row_mask,
                       TP* __restrict__ phi, int64_t rows, int H, int d, int D, float scale) {
  extern __shared__ __align__(16) float fm_smem[];
  constexpr int kFmI = 4, kFmRows = 16 * kFmI;
  const FmSmem s = fm_carve(fm_smem, kFmRows, D, d);
  const int h = blockIdx.y, rg = threadIdx.x >> 4, cg = (threadIdx.x & 15) * 4;
  const float* wh = w + (size_t)h * D * d;
  for (int i = threadIdx.x; i < D * d; i += kFmThreads) s.Wt[(i % d) * (D + 4) + i / d] = wh[i];
  const int64_t ntiles = (rows + kFmRows - 1) / kFmRows;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t row0 = tile * kFmRows;
    __syncthreads();
    fm_load_rows<kFmI>(s, x, row0, rows, H, h, d);
    __syncthreads();
    for (int col = cg; col < D; col += 64) {
      float u[kFmI][4];
      fm_product(u, s.X, d + 4, s.Wt, D + 4, d, rg, col);
#pragma unroll
      for (int i = 0; i < kFmI; ++i) {
        const int64_t row = row0 + rg + 16 * i;
        if (row >= rows) continue;
        const float sc = (row_mask && row_mask[row]) ? 0.f : scale;     // a masked row gets all-zero features
        float4 sn, cs;
        fm_sincos(u[i][0], sn.x, cs.x); fm_sincos(u[i][1], sn.y, cs.y); fm_sincos(u[i][2], sn.z, cs.z); fm_sincos(u[i][3], sn.w, cs.w);
        TP* dst = phi + ((size_t)row * H + h) * 2 * D + col;
        store4(dst, make_float4(sn.x * sc, sn.y * sc, sn.z * sc, sn.w * sc));
        store4(dst + D, make_float4(cs.x * sc, cs.y * sc, cs.z * sc, cs.w * sc));
      }
    }
  }
}

// Backward.  With g_u = scale * (g_sin * cos u - g_cos * sin u):
//   g_xh = W^T g_u;  g_x = g_xh / (n + eps) - xh * (xh . g_xh) / n;  g_W += g_u (x) xh
// GWT: 4 x 4 tiles of g_W per thread (D d <= 4096 GWT), summed per 64 rows from zero and kept in registers over the tiles.
template <typename T, int GWT, int NI>
__global__ void __launch_bounds__(kFmThreads, GWT == 1 ? 2 : 1)
feature_map_bwd_kernel(const T* __restrict__ x, const float* __restrict__ w, const uint8_t* __restrict__ row_mask,
                       const T* __restrict__ g_phi, T* __restrict__ g_x, float* __restrict__ g_w,
                       int64_t rows, int H, int d, int D, float scale) {
  extern __shared__ __align__(16) float fm_smem[];
  constexpr int kFmI = NI, kFmRows = 16 * NI;
  const FmSmem s = fm_carve(fm_smem, kFmRows, D, d);
  const int h = blockIdx.y, rg = threadIdx.x >> 4, cg = (threadIdx.x & 15) * 4;
  const float* wh = w + (size_t)h * D * d;
  for (int i = threadIdx.x; i < D * d; i += kFmThreads) {
    const int j = i / d, l = i - j * d;
    s.Wt[l * (D + 4) + j] = s.W[j * (d + 4) + l] = wh[i];
  }
  float gw[GWT][16];
#pragma unroll
  for (int k = 0; k < GWT; ++k)
#pragma unroll
    for (int e = 0; e < 16; ++e) gw[k][e] = 0.f;
  const int wt = d / 4, ntw = g_w ? (D / 4) * wt : 0;
  const int64_t ntiles = (rows + kFmRows - 1) / kFmRows;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t row0 = tile * kFmRows;
    __syncthreads();
    fm_load_rows<kFmI>(s, x, row0, rows, H, h, d);
    __syncthreads();
    float dot[kFmI];
#pragma unroll
    for (int i = 0; i < kFmI; ++i) dot[i] = 0.f;
    for (int col = cg; col < D; col += 64) {
      float u[kFmI][4];
      float4 gs[kFmI], gc[kFmI];                              // asked for before the product, which their flight hides
#pragma unroll
      for (int i = 0; i < kFmI; ++i) {
        const int64_t row = row0 + rg + 16 * i;
        const bool live = row < rows && !(row_mask && row_mask[row]);     // a masked row's features are constants: no gradient
        const T* gp = g_phi + ((size_t)row * H + h) * 2 * D + col;
        gs[i] = live ? load4(gp) : make_float4(0.f, 0.f, 0.f, 0.f);
        gc[i] = live ? load4(gp + D) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      fm_product(u, s.X, d + 4, s.Wt, D + 4, d, rg, col);
#pragma unroll
      for (int i = 0; i < kFmI; ++i) {
        float4 gu;
        float sn, cs;
        fm_sincos(u[i][0], sn, cs); gu.x = scale * (gs[i].x * cs - gc[i].x * sn);
        fm_sincos(u[i][1], sn, cs); gu.y = scale * (gs[i].y * cs - gc[i].y * sn);
        fm_sincos(u[i][2], sn, cs); gu.z = scale * (gs[i].z * cs - gc[i].z * sn);
        fm_sincos(u[i][3], sn, cs); gu.w = scale * (gs[i].w * cs - gc[i].w * sn);
        dot[i] = fmaf(gu.x, u[i][0], fmaf(gu.y, u[i][1], fmaf(gu.z, u[i][2], fmaf(gu.w, u[i][3], dot[i]))));
        store4(s.GU + (rg + 16 * i) * (D + 4) + col, gu);
      }
    }
#pragma unroll
    for (int i = 0; i < kFmI; ++i) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) dot[i] += __shfl_xor_sync(0xffffffffu, dot[i], o);
      if (cg == 0) s.c2[rg + 16 * i] = dot[i];
    }
    __syncthreads();
    for (int col = cg; col < d; col += 64) {
      float gx[kFmI][4];
      fm_product(gx, s.GU, D + 4, s.W, d + 4, D, rg, col);
#pragma unroll
      for (int i = 0; i < kFmI; ++i) {
        const int r = rg + 16 * i;
        const int64_t row = row0 + r;
        if (row >= rows) continue;
        const float n = s.nrm[r], inv = 1.f / (n + kNormEps), c2 = n > 0.f ? s.c2[r] / n : 0.f;
        const float4 xh = load4(s.X + r * (d + 4) + col);
        store4(g_x + ((size_t)row * H + h) * d + col, make_float4(gx[i][0] * inv - xh.x * c2, gx[i][1] * inv - xh.y * c2,
                                                                  gx[i][2] * inv - xh.z * c2, gx[i][3] * inv - xh.w * c2));
      }
    }
#pragma unroll
    for (int k = 0; k < GWT; ++k) {
      const int id = threadIdx.x + k * kFmThreads;
      if (id < ntw) {
        const float *pa = s.GU + (id / wt) * 4, *pb = s.X + (id % wt) * 4;
        float acc[4][4] = {};
#pragma unroll 4
        for (int r = 0; r < kFmRows; ++r) {
          const float4 a = load4(pa + r * (D + 4)), b = load4(pb + r * (d + 4));
          fm_axpy(acc[0], a.x, b); fm_axpy(acc[1], a.y, b); fm_axpy(acc[2], a.z, b); fm_axpy(acc[3], a.w, b);
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) gw[k][e] += acc[e >> 2][e & 3];
      }
    }
  }
  float* gwh = g_w ? g_w + (size_t)h * D * d : nullptr;
#pragma unroll
  for (int k = 0; k < GWT; ++k) {
    const int id = threadIdx.x + k * kFmThreads;
    if (id < ntw)
#pragma unroll
      for (int e = 0; e < 16; ++e) atomicAdd(gwh + ((id / wt) * 4 + (e >> 2)) * d + (id % wt) * 4 + (e & 3), gw[k][e]);
  }
}

// tensor-core forward for fp16 rows with head_dim = proj_dim = 64 (feature_map_tc.cu)
int launch_feature_map_fwd_tc(const __half* x, const float* w, const uint8_t* row_mask, __half* phi, const __half* x2,
                              const uint8_t* row_mask2, __half* phi2, int64_t rows, int H, float scale, int sms, cudaStream_t st);
int launch_feature_map_bwd_tc(const __half* x, const float* w, const uint8_t* row_mask, const __half* g_phi, __half* g_x,
                              const __half* x2, const uint8_t* row_mask2, const __half* g_phi2, __half* g_x2, float* g_w,
                              int64_t rows, int H, float scale, int sms, cudaStream_t st);

// split operands on the tensor cores for widths up to 64 (feature_map_mma.cu)
template <typename TX, typename TP>
int launch_feature_map_mma_fwd(const TX* x, const float* w, const uint8_t* row_mask, TP* phi, int64_t rows, int H, int d, int D, float scale,
                               int sms, cudaStream_t st);
template <typename T>
int launch_feature_map_mma_bwd(const T* x, const float* w, const uint8_t* row_mask, const T* g_phi, T* g_x, float* g_w, int64_t rows, int H,
                               int d, int D, float scale, int sms, cudaStream_t st);

static int fm_check(const void* x, const float* w, int64_t rows, int H, int d, int D) {
  RFA_REQUIRE(x && w, RFA_EINVAL, "feature_map: null pointer");
  RFA_REQUIRE(rows >= 0 && H > 0 && d > 0 && D > 0, RFA_EINVAL, "feature_map: rows=%lld H=%d d=%d D=%d",
              (long long)rows, H, d, D);
  RFA_REQUIRE(d % 8 == 0 && D % 8 == 0 && d <= 128 && D <= 128, RFA_EUNSUPPORTED,
              "feature_map: need d%%8==0, D%%8==0, d<=128, D<=128 (got d=%d D=%d)", d, D);
  RFA_REQUIRE(H <= 65535, RFA_EUNSUPPORTED, "feature_map: H=%d exceeds 65535", H);
  return 0;
}

// Whether the tensor-core kernels take it: a warp of theirs owns 16 rows, and below four of those to an SM its chain through
// products and sines is longer than what the register tiles here take with a whole CTA to 64 (32) rows.  us, here / there: fp32 64 x 64,
// 8 heads x 16, 256, 1024, 1536, 2048, 3072 rows forward 6.1 / 7.0, 7.3 / 7.1, 7.4 / 8.1, 10.2 / 8.4, 10.2 / 8.4, 13.6 / 10.4, backward
// 10.5 / 14.1, 10.8 / 14.7, 16.4 / 18.0, 21.5 / 18.7, 22.5 / 19.4, 37.3 / 22.4; 32 x 32, 16 x 512 5.9 / 5.6 and 9.9 / 10.6, 8 x 1536 7.2 / 5.8
// and 13.6 / 11.3.
// The line is higher
//  - where D > 32 and d <= 32, as the products are a small part there: 64 x 8, 16 heads x 600, 900, 1300 rows forward 5.7 / 7.0, 5.7 / 7.2, 7.2 / 7.7,
//    64 heads x 500 9.0 / 8.8; backward 13.1 / 13.2, 13.6 / 13.8, 22.1 / 14.9;
//  - for the backward of few heads, whose CTAs all add to the same matrices: 64 x 64, 1 head x 9600, 14400, 20800 rows 21.2 / 24.7, 24.1 / 25.5, 32.6 / 26.7;
//  - where the heads are more than the CTAs that the SMs hold, each of which has W to split: 64 x 64, 400 heads x 24, 52, 80 rows forward 12.1 / 15.0,
//    13.1 / 14.9, 21.6 / 15.7, 64 x 8, 400 heads x 160 17.0 / 21.3.
static bool fm_mma(int64_t rows, int H, int d, int D, int sms, bool backward) {
  if (d > 64 || D > 64) return false;
  const bool lean = D > 32 && d <= 32;
  const int64_t a_head = (rows + 15) / 16, line = lean ? (backward ? 8 : 12) : backward && H < 8 ? 8 : 4;
  return a_head * H > line * sms && (H <= 2 * sms || a_head >= (lean && !backward ? 32 : 5));
}

// CTAs per head, so that the grid is one wave of the `ctas` that an SM holds
static int fm_grid_x(int64_t rows, int tile, int H, int ctas) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t ntiles = (rows + tile - 1) / tile, fit = (int64_t)ctas * sms / H, want = fit < 1 ? 1 : fit;
  return (int)(ntiles < want ? ntiles : want);
}
static int fm_ctas(size_t smem, int most) {
  const int n = (int)(227 * 1024 / (smem + 1024));
  return n < 1 ? 1 : n < most ? n : most;
}

}  // namespace rfa

using namespace rfa;

extern "C" int rfa_feature_map_fwd_masked(const void* x, int x_dtype, const float* w, const uint8_t* row_mask, void* phi,
                                          int phi_dtype, int64_t rows, int H, int d, int D, float scale, rfa_stream_t stream) {
  if (int e = fm_check(x, w, rows, H, d, D)) return e;
  RFA_REQUIRE(phi, RFA_EINVAL, "feature_map_fwd: null output");
  RFA_REQUIRE(aligned16(x) && aligned16(w) && aligned16(phi), RFA_EALIGN, "feature_map_fwd: 16-byte alignment required");
  if (rows == 0) return 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (x_dtype == RFA_F16 && phi_dtype == RFA_F16 && d == 64 && D == 64)
    return launch_feature_map_fwd_tc((const __half*)x, w, row_mask, (__half*)phi, nullptr, nullptr, nullptr, rows, H, scale, sms,
                                     as_stream(stream));
  if (fm_mma(rows, H, d, D, sms, false)) {
#define RFA_MMA(TX, TP) return launch_feature_map_mma_fwd<TX, TP>((const TX*)x, w, row_mask, (TP*)phi, rows, H, d, D, scale, sms, as_stream(stream))
    if (x_dtype == RFA_F16 && phi_dtype == RFA_F16) RFA_MMA(__half, __half);
    if (x_dtype == RFA_F32 && phi_dtype == RFA_F32) RFA_MMA(float, float);
    if (x_dtype == RFA_F16 && phi_dtype == RFA_F32) RFA_MMA(__half, float);
    if (x_dtype == RFA_F32 && phi_dtype == RFA_F16) RFA_MMA(float, __half);
#undef RFA_MMA
  }
  const size_t smem = fm_smem_floats(64, D, d, false) * sizeof(float);      // 100 KB at most (D, d <= 128)
  const dim3 grid(fm_grid_x(rows, 64, H, fm_ctas(smem, 4)), H);
  cudaStream_t st = as_stream(stream);
#define RFA_LAUNCH(TX, TP)                                                                         \
  do {                                                                                             \
    cudaFuncSetAttribute(feature_map_fwd_kernel<TX, TP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    feature_map_fwd_kernel<TX, TP><<<grid, kFmThreads, smem, st>>>((const TX*)x, w, row_mask, (TP*)phi, rows, H, d, D, scale); \
  } while (0)
  if (x_dtype == RFA_F16 && phi_dtype == RFA_F16) RFA_LAUNCH(__half, __half);
  else if (x_dtype == RFA_F32 && phi_dtype == RFA_F32) RFA_LAUNCH(float, float);
  else if (x_dtype == RFA_F16 && phi_dtype == RFA_F32) RFA_LAUNCH(__half, float);
  else if (x_dtype == RFA_F32 && phi_dtype == RFA_F16) RFA_LAUNCH(float, __half);
  else return fail(RFA_EUNSUPPORTED, "feature_map_fwd: bad dtype %d/%d", x_dtype, phi_dtype);
#undef RFA_LAUNCH
  return check_launch("rfa_feature_map_fwd");
}

extern "C" int rfa_feature_map_fwd(const void* x, int x_dtype, const float* w, void* phi, int phi_dtype,
                                   int64_t rows, int H, int d, int D, float scale, rfa_stream_t stream) {
  return rfa_feature_map_fwd_masked(x, x_dtype, w, nullptr, phi, phi_dtype, rows, H, d, D, scale, stream);
}

extern "C" int rfa_feature_map_bwd_masked(const void* x, int x_dtype, const float* w, const uint8_t* row_mask, const void* g_phi,
                                          int g_dtype, void* g_x, int gx_dtype, float* g_w, int64_t rows, int H, int d, int D,
                                          float scale, rfa_stream_t stream) {
  if (int e = fm_check(x, w, rows, H, d, D)) return e;
  RFA_REQUIRE(g_phi && g_x, RFA_EINVAL, "feature_map_bwd: null pointer");
  RFA_REQUIRE(aligned16(x) && aligned16(w) && aligned16(g_phi) && aligned16(g_x) && aligned16(g_w), RFA_EALIGN,
              "feature_map_bwd: 16-byte alignment required");
  RFA_REQUIRE(x_dtype == g_dtype && x_dtype == gx_dtype, RFA_EUNSUPPORTED,
              "feature_map_bwd: x, g_phi and g_x must share one dtype");
  if (rows == 0) return 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (x_dtype == RFA_F16 && d == 64 && D == 64)
    return launch_feature_map_bwd_tc((const __half*)x, w, row_mask, (const __half*)g_phi, (__half*)g_x, nullptr, nullptr, nullptr,
                                     nullptr, g_w, rows, H, scale, sms, as_stream(stream));
  if (fm_mma(rows, H, d, D, sms, true)) {
    if (x_dtype == RFA_F16) return launch_feature_map_mma_bwd((const __half*)x, w, row_mask, (const __half*)g_phi, (__half*)g_x, g_w, rows, H, d, D,
                                                              scale, sms, as_stream(stream));
    if (x_dtype == RFA_F32) return launch_feature_map_mma_bwd((const float*)x, w, row_mask, (const float*)g_phi, (float*)g_x, g_w, rows, H, d, D,
                                                              scale, sms, as_stream(stream));
  }
  const bool small = D * d <= 4096;
  // Tiles of 32 rows where those of 64 would not give every SM one: a tile's three products follow one another, and so few
  // CTAs are bound by that chain.  (128 x 128, 8 heads x 1, 64, 512 rows: 39, 42, 43 us in
  // tiles of 64, 29, 30, 33 in tiles of 32; 64 x 64, 8 heads x 256 rows: 14.8 and 11.0.)
  const int tile = (rows + 63) / 64 * H < sms ? 32 : 64;
  const size_t smem = fm_smem_floats(tile, D, d, true) * sizeof(float);      // 199 KB at most (64 rows, D, d <= 128)
  const dim3 grid(fm_grid_x(rows, tile, H, fm_ctas(smem, small ? 2 : 1)), H);
  cudaStream_t st = as_stream(stream);
#define RFA_LAUNCH1(T, GWT, NI)                                                                    \
  do {                                                                                             \
    cudaFuncSetAttribute(feature_map_bwd_kernel<T, GWT, NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    feature_map_bwd_kernel<T, GWT, NI><<<grid, kFmThreads, smem, st>>>((const T*)x, w, row_mask, (const T*)g_phi, (T*)g_x, g_w, rows, H, d, \
                                                                   D, scale);                      \
  } while (0)
#define RFA_LAUNCH2(T, GWT) do { if (tile == 32) RFA_LAUNCH1(T, GWT, 2); else RFA_LAUNCH1(T, GWT, 4); } while (0)
#define RFA_LAUNCH(T) do { if (small) RFA_LAUNCH2(T, 1); else RFA_LAUNCH2(T, 4); } while (0)
  if (x_dtype == RFA_F16) RFA_LAUNCH(__half);
  else if (x_dtype == RFA_F32) RFA_LAUNCH(float);
  else return fail(RFA_EUNSUPPORTED, "feature_map_bwd: bad dtype %d", x_dtype);
#undef RFA_LAUNCH
#undef RFA_LAUNCH1
#undef RFA_LAUNCH2
  return check_launch("rfa_feature_map_bwd");
}

extern "C" int rfa_feature_map_bwd(const void* x, int x_dtype, const float* w, const void* g_phi, int g_dtype,
                                   void* g_x, int gx_dtype, float* g_w, int64_t rows, int H, int d, int D,
                                   float scale, rfa_stream_t stream) {
  return rfa_feature_map_bwd_masked(x, x_dtype, w, nullptr, g_phi, g_dtype, g_x, gx_dtype, g_w, rows, H, d, D, scale, stream);
}

// The feature maps of two arrays of one shape that share W (q and k of a self-attention layer) in one launch: one ramp
// and one W tile instead of two, and in the backward one g_W accumulator for both.  fp16, head_dim = proj_dim = 64 only
// (RFA_EUNSUPPORTED otherwise: call the single-array entry points twice).
extern "C" int rfa_feature_map_fwd_pair(const void* x_a, const void* x_b, const float* w, const uint8_t* row_mask_a,
                                        const uint8_t* row_mask_b, void* phi_a, void* phi_b, int64_t rows, int H, int d, int D,
                                        float scale, rfa_stream_t stream) {
  if (int e = fm_check(x_a, w, rows, H, d, D)) return e;
  RFA_REQUIRE(d == 64 && D == 64, RFA_EUNSUPPORTED, "feature_map_fwd_pair: built for head_dim = proj_dim = 64, fp16 (got %d, %d)", d, D);
  RFA_REQUIRE(rows == 0 || (x_b && phi_a && phi_b), RFA_EINVAL, "feature_map_fwd_pair: null pointer");
  RFA_REQUIRE(aligned16(x_a) && aligned16(x_b) && aligned16(w) && aligned16(phi_a) && aligned16(phi_b), RFA_EALIGN,
              "feature_map_fwd_pair: 16-byte alignment required");
  if (rows == 0) return 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return launch_feature_map_fwd_tc((const __half*)x_a, w, row_mask_a, (__half*)phi_a, (const __half*)x_b, row_mask_b, (__half*)phi_b,
                                   rows, H, scale, sms, as_stream(stream));
}

extern "C" int rfa_feature_map_bwd_pair(const void* x_a, const void* x_b, const float* w, const uint8_t* row_mask_a,
                                        const uint8_t* row_mask_b, const void* g_phi_a, const void* g_phi_b, void* g_x_a,
                                        void* g_x_b, float* g_w, int64_t rows, int H, int d, int D, float scale,
                                        rfa_stream_t stream) {
  if (int e = fm_check(x_a, w, rows, H, d, D)) return e;
  RFA_REQUIRE(d == 64 && D == 64, RFA_EUNSUPPORTED, "feature_map_bwd_pair: built for head_dim = proj_dim = 64, fp16 (got %d, %d)", d, D);
  RFA_REQUIRE(rows == 0 || (x_b && g_phi_a && g_phi_b && g_x_a && g_x_b), RFA_EINVAL, "feature_map_bwd_pair: null pointer");
  RFA_REQUIRE(aligned16(x_a) && aligned16(x_b) && aligned16(w) && aligned16(g_phi_a) && aligned16(g_phi_b) && aligned16(g_x_a) &&
                  aligned16(g_x_b) && aligned16(g_w), RFA_EALIGN, "feature_map_bwd_pair: 16-byte alignment required");
  if (rows == 0) return 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return launch_feature_map_bwd_tc((const __half*)x_a, w, row_mask_a, (const __half*)g_phi_a, (__half*)g_x_a, (const __half*)x_b,
                                   row_mask_b, (const __half*)g_phi_b, (__half*)g_x_b, g_w, rows, H, scale, sms, as_stream(stream));
}

// ---------------------------------------------------------------------------
// Effective random matrices of a whole step in one launch: out[i] = sigma[i] * bank[idx[i]] * inv_tau[i]
// (upstream gathers the sampled matrices on the host, utils.py:62-87, and applies sigma / tau per layer with separate
// PyTorch ops, utils.py:90-97).  bank [n_bank, D, d] fp16 or fp32 stays resident on the device.
// ---------------------------------------------------------------------------
namespace rfa {
template <typename TB>
__global__ void gather_matrices_kernel(const TB* __restrict__ bank, int64_t n_bank, const int64_t* __restrict__ idx,
                                       const float* __restrict__ sigma, const float* __restrict__ inv_tau,
                                       float* __restrict__ out, int64_t n_out, int D, int d, int* __restrict__ bad) {
  const int64_t per = (int64_t)D * d;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n_out * per) return;
  const int64_t i = e / per, r = e % per;
  const int64_t src = idx[i];
  if (src < 0 || src >= n_bank) {          // a pick outside the bank: flag it and write zeros instead of reading out of bounds
    if (r == 0) atomicExch(bad, 1);
    out[e] = 0.f;
    return;
  }
  float w = to_f(bank[src * per + r]);
  if (sigma) w *= sigma[i * d + r % d];
  if (inv_tau) w *= inv_tau[i];
  out[e] = w;
}
}  // namespace rfa

extern "C" int rfa_gather_random_matrices(const void* bank, int bank_dtype, int64_t n_bank, const int64_t* idx, int64_t n_out,
                                          const float* sigma, const float* inv_tau, float* out, int D, int d, int* bad_index_flag,
                                          rfa_stream_t stream) {
  RFA_REQUIRE(bank && idx && out && bad_index_flag, RFA_EINVAL, "gather_random_matrices: null pointer");
  RFA_REQUIRE(n_bank > 0 && n_out >= 0 && D > 0 && d > 0, RFA_EINVAL, "gather_random_matrices: n_bank=%lld n_out=%lld D=%d d=%d",
              (long long)n_bank, (long long)n_out, D, d);
  RFA_REQUIRE(bank_dtype == RFA_F16 || bank_dtype == RFA_F32, RFA_EUNSUPPORTED, "gather_random_matrices: bank dtype %d", bank_dtype);
  if (n_out == 0) return 0;
  const int64_t total = n_out * D * d;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (bank_dtype == RFA_F16)
    gather_matrices_kernel<__half><<<blocks, 256, 0, as_stream(stream)>>>((const __half*)bank, n_bank, idx, sigma, inv_tau, out, n_out, D, d, bad_index_flag);
  else
    gather_matrices_kernel<float><<<blocks, 256, 0, as_stream(stream)>>>((const float*)bank, n_bank, idx, sigma, inv_tau, out, n_out, D, d, bad_index_flag);
  return check_launch("rfa_gather_random_matrices");
}
