// Feature map and its gradient for widths up to 64 that are not the fp16 64 x 64 of feature_map_tc.cu: fp32 rows, and fp16 rows of
// other widths (formulas in feature_map.cu).
//
// fp32 throughout, on the tensor cores: both operands of a product are split into two fp16 tiles under a power of two per block or row
// (generic_split.cuh; normalised rows are below 1 and share one), 22 bits each, and three mma.sync m16n8k16 make the product, lo hi,
// hi lo, hi hi; what is left out is 2^-22 of a term.  16 terms at a time from zero, those sums scaled and added in fp32.
// Register tiles on the FMA pipe (feature_map.cu) read 16 bytes of shared memory for every 8 FMAs, which bounded them, and the sines
// of CUDA's library are 75 instructions a pair (trig.cuh); splits into tf32 at every read (6 mma per 16 terms instead of 3, and 5
// instructions an element and read) were no faster than those.  What bounds it now is issue slots and fixed latencies at 16 warps an SM (slots
// 57 % forward, 49 % backward, no pipe above 33 %).
// fp32, 64 x 64, 4096 rows of 16 heads: forward 30.1 -> 18.2 us, backward 67.6 -> 41.8 (40.2 with one factor a block, 46.6 with faded rows in every one); 32 x 32, 4096 rows of 8 heads 11.8 -> 6.8 and 23.7 -> 14.4.
// Errors against fp64 (phi, g_x, g_W): 1.62, 2.27, 2.42e-7 -> 1.27, 1.72, 1.95e-7, from shorter chains of fp32 sums.
//
// A warp owns 16 rows: it loads, normalises and splits them, and their products, sines and results stay within the warp
// (accumulators of u are turned into g_u in registers, split into the warp's rows of a tile and multiplied by W again).  Only
// g_W = sum over rows needs the block: 8 warps take 16 x 32 of it each over all rows of the tile.
#include "generic_split.cuh"
#include "trig.cuh"

namespace rfa {
namespace fmm {

constexpr int kThreads = 256, kWarps = kThreads / 32, kMax = 64, kRows = 16 * kWarps;
constexpr int kP = kMax + 8;                        // pitch in halves: 8 rows start in 8 different 16-byte banks
constexpr float kXs = 16384.f, kXi = 1.f / kXs;     // the factor of normalised rows
constexpr uint32_t kW = 0, kX = kW + 2 * kMax * kP * 2, kWf = kX + 2 * kRows * kP * 2, kNrm = kWf + 16 * 4, kFwdBytes = kNrm + kRows * 4,
                   kG = kFwdBytes, kGf = kG + 2 * kRows * kP * 2, kBwdBytes = kGf + kRows * 4 * 4;
constexpr int kCtas = 2;                            // on an SM (three of the forward, at 80 registers a thread: 22.6 us instead of 18.2)
static_assert(kCtas * (kBwdBytes + 1024) <= 228 * 1024 && kG % 16 == 0, "feature_map_mma: shared memory");

__device__ __forceinline__ float2 both(float f) { return make_float2(f, f); }
// ---- products ------------------------------------------------------------------------------------------------------------------
// acc (16 x 32, nt blocks of 8 columns) = A B of two split operands, L terms: pa, pb the lane's shared-memory addresses of the first
// fragments, da, db their steps per 16 terms and dn B's per 16 columns, (TA, TB) whether the fragments are transposed; the sums over terms 16 l .. have
// the factors r(l), of rows g and g + 8, and f(l, n), of columns 16 n ..
template <bool TA, bool TB, class R, class F>
__device__ __forceinline__ void product(float (&acc)[4][4], int nt, int L, uint32_t pa, uint32_t a_lo, uint32_t da, uint32_t pb, uint32_t b_lo,
                                        uint32_t db, uint32_t dn, R r, F f) {
  gm_zero(acc);
#pragma unroll 1
  for (int l = 0; l < L; ++l, pa += da, pb += db) {
    const float2 fr = r(l);
    uint32_t ah[4], al[4];
    if (TA) { gm_ldsm_t(ah, pa); gm_ldsm_t(al, pa + a_lo); }
    else { gm_ldsm(ah, pa); gm_ldsm(al, pa + a_lo); }
#pragma unroll
    for (int n = 0; n < 2; ++n)
      if (2 * n < nt) {
        uint32_t bh[4], bl[4];
        if (TB) { gm_ldsm_t(bh, pb + n * dn); gm_ldsm_t(bl, pb + n * dn + b_lo); }
        else { gm_ldsm(bh, pb + n * dn); gm_ldsm(bl, pb + n * dn + b_lo); }
        float p[2][4];
        gm_mma16_0(p[0], al, bh[0], bh[1]);
        gm_mma16_0(p[1], al, bh[2], bh[3]);
        gm_mma16(p[0], ah, bl[0], bl[1]);
        gm_mma16(p[1], ah, bl[2], bl[3]);
        gm_mma16(p[0], ah, bh[0], bh[1]);
        gm_mma16(p[1], ah, bh[2], bh[3]);
        const float fn = f(l, n);
        const float2 sc = make_float2(fr.x * fn, fr.y * fn);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[2 * n + m][e] = fmaf(p[m][e], e < 2 ? sc.x : sc.y, acc[2 * n + m][e]);
      }
  }
}

// W_h in two parts, a warp per 16 x 16 block, zeros in its pad rows and columns
__device__ __forceinline__ void load_w(const GsSplit& W, const float* __restrict__ wh, int D, int d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int b = warp; b < 16; b += kWarps) {
    const int i0 = (b >> 2) * 16, j0 = (b & 3) * 16;
    if (i0 >= D || j0 >= d) continue;
    float a[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + g + 8 * r, j = j0 + 8 * n + 2 * t;
        const float2 v = i < D && j < d ? *reinterpret_cast<const float2*>(wh + i * d + j) : make_float2(0.f, 0.f);
        a[n][2 * r] = v.x; a[n][2 * r + 1] = v.y;
      }
    gs_put(W, i0, j0, a);
  }
}

// a warp's 16 rows: 16 lanes a row, all loads before the first use
template <typename T>
__device__ __forceinline__ void ask_rows(float4 (&v)[8], const T* __restrict__ x, int64_t row0, int64_t rows, int H, int h, int d, int lane) {
  const int c = (lane & 15) * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int64_t row = row0 + 2 * i + (lane >> 4);
    v[i] = row < rows && c < d ? load4(x + ((size_t)row * H + h) * d + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}
// normalised and split (columns up to the next multiple of 16: zeros from d on)
__device__ __forceinline__ void put_rows(const float4 (&v)[8], __half* hi, __half* lo, float* nrm, int d, int lane) {
  const int c = (lane & 15) * 4;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, v[i].w * v[i].w)));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float n = sqrtf(ss), inv = 1.f / (n + kNormEps);
    const int r = 2 * i + (lane >> 4);
    uint2 h, l;
    gs_parts<false>(v[i].x * inv, v[i].y * inv, kXs, h.x, l.x);
    gs_parts<false>(v[i].z * inv, v[i].w * inv, kXs, h.y, l.y);
    if (c < gm_round16(d)) {
      *reinterpret_cast<uint2*>(hi + r * kP + c) = h;
      *reinterpret_cast<uint2*>(lo + r * kP + c) = l;
    }
    if (c == 0) nrm[r] = n;
  }
}
__device__ __forceinline__ void store2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void store2(__half* p, float a, float b) { *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b); }
__device__ __forceinline__ float2 load2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load2(const __half* p) { return __half22float2(*reinterpret_cast<const __half2*>(p)); }

// grid (gx, H): a CTA takes an even share of its head's groups of 16 rows, eight at a time
struct Share { int64_t at, end; };
__device__ __forceinline__ Share share_of(int64_t rows) {
  const int64_t units = (rows + 15) / 16;
  return Share{units * blockIdx.x / gridDim.x, units * (blockIdx.x + 1) / gridDim.x};
}
struct Tiles {
  GsSplit W;                // [j][l]
  __half *xh, *xl;          // normalised rows
  GsByRow G;                // g_u [row][j]
  float* nrm;
};
__device__ __forceinline__ Tiles tiles_at(unsigned char* base) {
  Tiles s;
  s.W = GsSplit{(__half*)(base + kW), (__half*)(base + kW) + kMax * kP, (float*)(base + kWf), kP, 4};
  s.G = GsByRow{(__half*)(base + kG), (__half*)(base + kG) + kRows * kP, (float*)(base + kGf), kP, 4, 1};
  s.xh = (__half*)(base + kX); s.xl = s.xh + kRows * kP;
  s.nrm = (float*)(base + kNrm);
  return s;
}
// u = X W^T for columns 32 c .. 32 c + 31 of the rows from `row` of the tile
__device__ __forceinline__ void project(float (&u)[4][4], int nt, const Tiles& s, int row, int c, int d, int lane) {
  const float* f = s.W.inv_s + 2 * c * 4;
  product<false, false>(u, nt, (d + 15) / 16, gm_addr(s.xh + row * kP + gm_off_a(lane, kP)), 2 * kRows * kP, 32,
                        gm_addr(s.W.hi + 32 * c * kP + gm_off_b(lane, kP)), 2 * kMax * kP, 32, 32 * kP, [](int) { return both(kXi); }, [&](int l, int n) { return f[n * 4 + l]; });
}

// g_u.  g_x = g_u W is a product for each row by itself, so that a row must not lose bits to a larger one beside it: where a row of a block is
// below 2^-kEven of another, each has a factor of its own there (2^-27 of the row's largest element is the most that a shared one costs it).  g_W sums
// over rows, where one factor a block is what can be taken out of the sum: such blocks are split again for it (even_rows).
constexpr uint32_t kEven = 12;
static __device__ __noinline__ bool put_g_faded(GsByRow m, int r0, int j0, float4 x, float4 y, uint32_t line) {
  const float a[2][4] = {{x.x, x.y, x.z, x.w}, {y.x, y.y, y.z, y.w}};
  uint32_t mag[2];
  gs_row_mags<true>(mag, a);
  const bool own = __any_sync(0xffffffffu, mag[0] - 1 < line || mag[1] - 1 < line);      // 0 is not: it has no bits to lose
  if (!own) mag[0] = mag[1] = __reduce_max_sync(0xffffffffu, max(mag[0], mag[1]));
  gs_put_rows_as<true>(m, r0, j0, a, mag);
  return own;
}
// -> whether the block's rows have factors of their own
__device__ __forceinline__ bool put_g(const GsByRow& m, int r0, int j0, const float (&a)[2][4]) {
  uint32_t mag[2] = {0, 0};                            // this lane's part of a row: one that has not faded in any lane has not faded
#pragma unroll
  for (int e = 0; e < 8; ++e) mag[e >> 1 & 1] = max(mag[e >> 1 & 1], gs_mag(a[e >> 2][e & 3]));
  const uint32_t most = __reduce_max_sync(0xffffffffu, max(mag[0], mag[1])), exponent = most & kGsInf;
  const uint32_t line = most >= kGsInf ? ~0u : exponent > (kEven << 23) ? exponent - (kEven << 23) : 0u;
  if (__any_sync(0xffffffffu, mag[0] - 1 < line || mag[1] - 1 < line))
    return put_g_faded(m, r0, j0, make_float4(a[0][0], a[0][1], a[0][2], a[0][3]), make_float4(a[1][0], a[1][1], a[1][2], a[1][3]), line);
  const uint32_t all[2] = {most, most};
  gs_put_rows_as<false>(m, r0, j0, a, all);
  return false;
}
// the warp's blocks (bits of `own`) of finite numbers with one factor each again
static __device__ __noinline__ void even_rows(GsByRow m, int r0, uint32_t own) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int b = 0; b < 4; ++b) {
    if (!(own >> b & 1)) continue;
    float a[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) a[n][e] = gs_at(m, r0 + g + 8 * (e >> 1), 16 * b + 8 * n + 2 * t + (e & 1));
    uint32_t mag[2];
    gs_row_mags<false>(mag, a);
    mag[0] = mag[1] = __reduce_max_sync(0xffffffffu, max(mag[0], mag[1]));
    gs_put_rows_as<false>(m, r0, 16 * b, a, mag);      // every lane has read what it writes; the factors were read before the reduction
  }
}

template <typename TX, typename TP>
__global__ void __launch_bounds__(kThreads, kCtas)
feature_map_mma_fwd_kernel(const TX* __restrict__ x, const float* __restrict__ w, const uint8_t* __restrict__ row_mask, TP* __restrict__ phi,
                           int64_t rows, int H, int d, int D, float scale) {
  extern __shared__ __align__(16) unsigned char fmm_smem[];
  const Tiles s = tiles_at(fmm_smem);
  const int h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, r0 = warp * 16;
  const Share sh = share_of(rows);
  float4 v[8];
  ask_rows(v, x, (sh.at + warp) * 16, sh.at + warp < sh.end ? rows : 0, H, h, d, lane);
  load_w(s.W, w + (size_t)h * D * d, D, d);
  __syncthreads();
  for (int64_t unit = sh.at + warp; unit < sh.end; unit += kWarps) {
    __syncwarp();
    put_rows(v, s.xh + r0 * kP, s.xl + r0 * kP, s.nrm + r0, d, lane);
    __syncwarp();
    if (unit + kWarps < sh.end) ask_rows(v, x, (unit + kWarps) * 16, rows, H, h, d, lane);
    const int64_t row = unit * 16 + g;
    const float sc[2] = {row_mask && row < rows && row_mask[row] ? 0.f : scale, row_mask && row + 8 < rows && row_mask[row + 8] ? 0.f : scale};
    TP* dst = phi + ((size_t)row * H + h) * 2 * D + 2 * t;      // a masked row gets all-zero features
#pragma unroll 1
    for (int c = 0; 32 * c < D; ++c, dst += 32) {
      const int nt = min(4, D / 8 - 4 * c);
      float u[4][4];
      project(u, nt, s, r0, c, d, lane);
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (n < nt)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            float s0, c0, s1, c1;
            fm_sincos(u[n][2 * r], s0, c0);
            fm_sincos(u[n][2 * r + 1], s1, c1);
            if (row + 8 * r < rows) {
              TP* p = dst + (size_t)8 * r * H * 2 * D + 8 * n;
              store2(p, s0 * sc[r], s1 * sc[r]);
              store2(p + D, c0 * sc[r], c1 * sc[r]);
            }
          }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads, kCtas)
feature_map_mma_bwd_kernel(const T* __restrict__ x, const float* __restrict__ w, const uint8_t* __restrict__ row_mask,
                           const T* __restrict__ g_phi, T* __restrict__ g_x, float* __restrict__ g_w, int64_t rows, int H, int d, int D,
                           float scale) {
  extern __shared__ __align__(16) unsigned char fmm_smem[];
  const Tiles s = tiles_at(fmm_smem);
  const int h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, r0 = warp * 16;
  const float* wh = w + (size_t)h * D * d;
  const Share sh = share_of(rows);
  // this warp's part of g_W: rows j0 .., columns l0 ..
  const int j0 = (warp >> 1) * 16, l0 = (warp & 1) * 32, lt = g_w && j0 < D ? max(0, min(4, (d - l0 + 7) / 8)) : 0;
  float gw[4][4] = {};
  float4 v[8];
  ask_rows(v, x, (sh.at + warp) * 16, sh.at + warp < sh.end ? rows : 0, H, h, d, lane);
  load_w(s.W, wh, D, d);
  for (int64_t at = sh.at; at < sh.end; at += kWarps) {
    const int active = (int)min((int64_t)kWarps, sh.end - at);
    __syncthreads();                                  // W is there; the tile before has been read
    bool odd = false;
    uint32_t own = 0;                                 // blocks of g_u whose rows have factors of their own
    if (warp < active) {
      put_rows(v, s.xh + r0 * kP, s.xl + r0 * kP, s.nrm + r0, d, lane);
      __syncwarp();
      float dot[2] = {0.f, 0.f};
      const int64_t row = (at + warp) * 16 + g;
      const T* gp[2];
      bool live[2];                                   // a masked row's features are constants: no gradient
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        live[r] = row + 8 * r < rows && !(row_mask && row_mask[row + 8 * r]);
        gp[r] = g_phi + ((size_t)(row + 8 * r) * H + h) * 2 * D + 2 * t;
      }
#pragma unroll 1
      for (int c = 0; 32 * c < D; ++c) {
        const int nt = min(4, D / 8 - 4 * c);
        float2 gs[4][2], gc[4][2];                    // asked for before the product, which their flight hides
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const bool l = live[r] && n < nt;
            gs[n][r] = l ? load2(gp[r] + 32 * c + 8 * n) : make_float2(0.f, 0.f);
            gc[n][r] = l ? load2(gp[r] + 32 * c + 8 * n + D) : make_float2(0.f, 0.f);
          }
        float u[4][4];
        project(u, nt, s, r0, c, d, lane);
#pragma unroll
        for (int b = 0; b < 2; ++b)
          if (2 * b < nt) {
            float a[2][4];
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const int n = 2 * b + m;
                float sn, cs;
                fm_sincos(u[n][2 * r], sn, cs);
                const float e = scale * (gs[n][r].x * cs - gc[n][r].x * sn);
                fm_sincos(u[n][2 * r + 1], sn, cs);
                const float f = scale * (gs[n][r].y * cs - gc[n][r].y * sn);
                a[m][2 * r] = n < nt ? e : 0.f; a[m][2 * r + 1] = n < nt ? f : 0.f;      // (a block's second half may lie past D)
                dot[r] = fmaf(a[m][2 * r], n < nt ? u[n][2 * r] : 0.f, fmaf(a[m][2 * r + 1], n < nt ? u[n][2 * r + 1] : 0.f, dot[r]));
                odd |= !(fabsf(a[m][2 * r]) < CUDART_INF_F) | !(fabsf(a[m][2 * r + 1]) < CUDART_INF_F);
              }
            own |= (uint32_t)put_g(s.G, r0, 32 * c + 16 * b, a) << (2 * c + b);
          }
      }
      float c2[2], inv[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        dot[r] = gm_quad(dot[r]);
        const float n = s.nrm[r0 + g + 8 * r];
        inv[r] = 1.f / (n + kNormEps);
        c2[r] = n > 0.f ? dot[r] / n : 0.f;
      }
      const bool scalar = __any_sync(0xffffffffu, odd);
      __syncwarp();
#pragma unroll 1
      for (int c = 0; 32 * c < d; ++c) {
        const int nt = min(4, d / 8 - 4 * c);
        float a[4][4];
        if (scalar) {                                 // inf times the two parts of a number may be inf - inf
#pragma unroll
          for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              a[n][e] = 0.f;
              if (n < nt)
#pragma unroll 1
                for (int j = 0; j < D; ++j) a[n][e] = fmaf(gs_at(s.G, r0 + g + 8 * (e >> 1), j), wh[j * d + 32 * c + 8 * n + 2 * t + (e & 1)], a[n][e]);
            }
        } else {
          const float *fg = s.G.inv_s + (r0 + g) * 4, *fw = s.W.inv_s + 2 * c;
          product<false, true>(a, nt, (D + 15) / 16, gm_addr(s.G.hi + r0 * kP + gm_off_a(lane, kP)), 2 * kRows * kP, 32,
                               gm_addr(s.W.hi + 32 * c + gm_off_a(lane, kP)), 2 * kMax * kP, 32 * kP, 32,
                               [&](int l) { return make_float2(fg[l], fg[32 + l]); }, [&](int l, int n) { return fw[4 * l + n]; });
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          if (row + 8 * r >= rows) continue;
          T* dst = g_x + ((size_t)(row + 8 * r) * H + h) * d + 32 * c + 2 * t;
          const int xo = (r0 + g + 8 * r) * kP + 32 * c + 2 * t;
#pragma unroll
          for (int n = 0; n < 4; ++n)
            if (n < nt) {
              const float2 fh = load2(s.xh + xo + 8 * n), fl = load2(s.xl + xo + 8 * n);
              store2(dst + 8 * n, a[n][2 * r] * inv[r] - (fh.x + fl.x) * kXi * c2[r], a[n][2 * r + 1] * inv[r] - (fh.y + fl.y) * kXi * c2[r]);
            }
        }
      }
      if (own && g_w && !scalar) even_rows(s.G, r0, own);
    }
    const bool scalar = __syncthreads_or(odd) != 0;
    if (warp < (int)min((int64_t)kWarps, sh.end - at - kWarps)) ask_rows(v, x, (at + kWarps + warp) * 16, rows, H, h, d, lane);
    if (lt > 0) {
      float a[4][4];
      const bool second = j0 + 8 < D;                 // D may end after the first 8 of this warp's 16 rows
      if (scalar) {
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            a[n][e] = 0.f;
            const int xo = l0 + 8 * n + 2 * t + (e & 1);
            if (n < lt && (e < 2 || second))
#pragma unroll 1
              for (int r = 0; r < 16 * active; ++r)
                a[n][e] = fmaf(gs_at(s.G, r, j0 + g + 8 * (e >> 1)), (__half2float(s.xh[r * kP + xo]) + __half2float(s.xl[r * kP + xo])) * kXi, a[n][e]);
          }
      } else {
        const float* fg = s.G.inv_s + (j0 >> 4);
        product<true, true>(a, lt, active, gm_addr(s.G.hi + j0 + gm_off_b(lane, kP)), 2 * kRows * kP, 32 * kP,
                            gm_addr(s.xh + l0 + gm_off_a(lane, kP)), 2 * kRows * kP, 32 * kP, 32, [&](int l) { return both(fg[64 * l]); }, [](int, int) { return kXi; });
      }
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) gw[n][e] += a[n][e];
    }
  }
  if (lt > 0 && sh.at < sh.end) {
    float* dst = g_w + ((size_t)h * D + j0 + g) * d + l0 + 2 * t;
#pragma unroll
    for (int n = 0; n < 4; ++n)
      if (n < lt)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (e < 2 || j0 + 8 < D) atomicAdd(dst + (e >> 1) * 8 * d + 8 * n + (e & 1), gw[n][e]);
  }
}

// CTAs per head: one wave of those that the SMs hold, none without rows
static int grid_x(int64_t rows, int H, int sms) {
  const int64_t units = (rows + 15) / 16, fit = (int64_t)kCtas * sms / H, want = fit < 1 ? 1 : fit;
  return (int)(units < want ? units : want);
}
template <class KERNEL, class... Args>
static int launch(KERNEL kernel, const char* what, dim3 grid, size_t smem, cudaStream_t st, Args... args) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail((int)e, "%s: cannot reserve %zu bytes of shared memory: %s", what, smem, cudaGetErrorString(e));
  kernel<<<grid, kThreads, smem, st>>>(args...);
  return check_launch(what);
}

}  // namespace fmm

template <typename TX, typename TP>
int launch_feature_map_mma_fwd(const TX* x, const float* w, const uint8_t* row_mask, TP* phi, int64_t rows, int H, int d, int D, float scale,
                               int sms, cudaStream_t st) {
  return fmm::launch(fmm::feature_map_mma_fwd_kernel<TX, TP>, "rfa_feature_map_fwd", dim3(fmm::grid_x(rows, H, sms), H), fmm::kFwdBytes, st, x, w,
                     row_mask, phi, rows, H, d, D, scale);
}
template <typename T>
int launch_feature_map_mma_bwd(const T* x, const float* w, const uint8_t* row_mask, const T* g_phi, T* g_x, float* g_w, int64_t rows, int H,
                               int d, int D, float scale, int sms, cudaStream_t st) {
  return fmm::launch(fmm::feature_map_mma_bwd_kernel<T>, "rfa_feature_map_bwd", dim3(fmm::grid_x(rows, H, sms), H), fmm::kBwdBytes, st, x, w, row_mask,
                     g_phi, g_x, g_w, rows, H, d, D, scale);
}
#define RFA_FMM_FWD(TX, TP) \
  template int launch_feature_map_mma_fwd<TX, TP>(const TX*, const float*, const uint8_t*, TP*, int64_t, int, int, int, float, int, cudaStream_t);
RFA_FMM_FWD(float, float) RFA_FMM_FWD(__half, __half) RFA_FMM_FWD(__half, float) RFA_FMM_FWD(float, __half)
#define RFA_FMM_BWD(T) \
  template int launch_feature_map_mma_bwd<T>(const T*, const float*, const uint8_t*, const T*, T*, float*, int64_t, int, int, int, float, int, cudaStream_t);
RFA_FMM_BWD(float) RFA_FMM_BWD(__half)

}  // namespace rfa
