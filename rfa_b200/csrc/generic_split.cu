// Causal RFA and the state reduction for geometries other than K = 128, d = 64, in chunks on the tensor cores: the ones whose state
// fits in shared memory twice (once in fp32, once as operand).  What does not fit is served by generic_mma.cu, whose formulas
// per chunk, segments and treatment of non-finite values these kernels share.
//
// State, weights and partial sums are fp32; as operands they are split into two fp16 tiles (generic_split.cuh), once, by the warp that
// made them.
// The kernels of generic_mma.cu split into tf32 in registers, at every read: 28 instructions a fragment of A, and four mma per 16 terms
// where there are two here.  Both are bound by issue slots and a chunk's chain of phases, not by memory or the tensor pipe (slots 50 %, ALU 35 %,
// tensor pipe 12 %, a third of a warp's wait at the chunk's barriers): forward + backward kernels 185 -> 137 us at (K, d) = (64, 32), 64 heads x
// 1024 tokens, 138 -> 90 at (96, 40), 64 x 300, 392 -> 317 at (128, 128), 64 x 512, 123 -> 57 at (128, 128), 8 x 200.
#include "generic_split.cuh"
#include "segments.cuh"
#include "sm100.cuh"

namespace rfa {

constexpr int kGsRegs = 80;      // 24 warps on an SM: three CTAs of 256 threads, two of 384 or one of 768
// Whether launches may be placed while the previous kernel drains: segments of at most four chunks.  A step is five to seven launches then, and
// their gaps a good part of it; longer kernels lose more to the CTAs' uneven placement than the gaps cost.  us a step without / with: (64, 32), 64
// heads x 1024 tokens (4 chunks) 145.4 / 136.2, 128 x 512 (4) 143.6 / 136.5; (96, 40), 64 x 300 (3) 96.8 / 90.2, 128 x 512 (8) 219 / 231; (128, 128),
// 64 x 512 (8) 322.8 / 320.5, 128 x 512 (16) 491 / 501.
__host__ __device__ inline bool gs_pdl(int64_t tseg, int C) { return tseg <= 4 * C; }

struct GsLayout {
  int Kp, dp, px, py, ps, ph, pc;      // K and d rounded up to 16; pitches of X tiles (q, k), Y tiles (v, g), the fp32 state, [.][d] and [C][C] split matrices
  uint32_t x_bytes, y_bytes;
  uint32_t S, z, s_hi, s_f, P, p_f, D, d_f, G, g_f, row, tile, total;
};
enum { kGsState = 1, kGsP = 2, kGsD = 4, kGsG = 8, kGsByRow = 16 };      // which split matrices a kernel holds; P with a factor a row
__host__ __device__ inline GsLayout gs_layout(int C, int K, int d, int nx, int ny, int has, int row_floats) {
  GsLayout L;
  L.Kp = gm_round16(K); L.dp = gm_round16(d);
  L.px = L.Kp + 8; L.py = d + 8; L.ps = d + 4; L.ph = L.dp + 8; L.pc = C + 8;
  L.x_bytes = (uint32_t)C * L.px * 2; L.y_bytes = (uint32_t)C * L.py * 2;
  uint32_t at = 0;
  auto take = [&](uint32_t bytes) { const uint32_t r = at; at += (bytes + 15) & ~15u; return r; };
  L.S = take((uint32_t)L.Kp * L.ps * 4);
  L.z = take((uint32_t)L.Kp * 4);
  L.s_hi = take(has & kGsState ? (uint32_t)L.Kp * L.ph * 4 : 0);
  L.s_f = take(has & kGsState ? (uint32_t)(L.Kp / 16) * (L.dp / 16) * 4 : 0);
  L.P = take(has & kGsP ? (uint32_t)C * L.pc * 4 : 0);
  L.p_f = take(has & kGsP ? (uint32_t)(C / 16) * (has & kGsByRow ? C : C / 16) * 4 : 0);
  L.D = take(has & kGsD ? (uint32_t)C * L.pc * 4 : 0);
  L.d_f = take(has & kGsD ? (uint32_t)(C / 16) * (C / 16) * 4 : 0);
  L.G = take(has & kGsG ? (uint32_t)C * L.ph * 4 : 0);
  L.g_f = take(has & kGsG ? (uint32_t)(C / 16) * L.dp * 2 : 0);
  L.row = take((uint32_t)row_floats * 4);
  L.tile = at;
  L.total = at + nx * L.x_bytes + ny * L.y_bytes;
  return L;
}
__device__ __forceinline__ GsSplit gs_split_at(unsigned char* base, uint32_t hi, uint32_t f, int rows, int pitch, int sp) {
  __half* p = (__half*)(base + hi);
  return GsSplit{p, p + rows * pitch, (float*)(base + f), pitch, sp};
}
// per-row floats of each kernel
__host__ __device__ inline int gs_rows_fwd(int C) { return (C / 16 + 1) * C; }                                  // rs, qz
__host__ __device__ inline int gs_rows_q(int C, int K) { return (2 * (C / 16) + gm_groups32(K) + 3) * C; }      // rs, pg, wq, qz, inv, gz
__host__ __device__ inline int gs_rows_w(int C) { return 3 * C + 16; }                                          // inv, gz, gz in two fp16 parts, its factors
__host__ __device__ inline GsLayout gs_layout_fwd(int C, int K, int d) { return gs_layout(C, K, d, 2, 1, kGsState | kGsP | kGsByRow, gs_rows_fwd(C)); }
__host__ __device__ inline GsLayout gs_layout_q(int C, int K, int d) { return gs_layout(C, K, d, 2, 2, kGsState | kGsD, gs_rows_q(C, K)); }
__host__ __device__ inline GsLayout gs_layout_kv(int C, int K, int d) { return gs_layout(C, K, d, 2, 2, kGsState | kGsP | kGsD | kGsG, gs_rows_w(C)); }
__host__ __device__ inline GsLayout gs_layout_state(int C, int K, int d, bool w) { return gs_layout(C, K, d, 1, 1, w ? kGsG : 0, w ? gs_rows_w(C) : 0); }

// ---- products ------------------------------------------------------------------------------------------------------------------
// acc (16 x 8 NT) += sum over l in [l0, l1) of A(i, l) B(l, j), B columns j0.. of an fp16 tile stored along j.  f: a lane's factors (rows g, g + 8) for
// the first 16 terms, df to the next
template <int NT, bool TRANS, class F>
__device__ __forceinline__ void gs_product(float (&acc)[NT][4], int nt, int l0, int l1, const __half* hi, const __half* lo_, int at, uint32_t da, GmTile y,
                                           int j0, F f) {
  const int lane = threadIdx.x & 31;
  uint32_t ph = gm_addr(hi + at), pb = gm_addr(y.p + j0 + gm_off_a(lane, y.pitch) + l0 * y.pitch);
  const uint32_t lo = (uint32_t)((const char*)lo_ - (const char*)hi), db = 32u * y.pitch;
#pragma unroll 1
  for (int l = l0; l < l1; l += 16, ph += da, pb += db) {
    uint32_t h[4], o[4];
    if (TRANS) { gm_ldsm_t(h, ph); gm_ldsm_t(o, ph + lo); }
    else { gm_ldsm(h, ph); gm_ldsm(o, ph + lo); }
    const float2 sc = f();
#pragma unroll
    for (int n = 0; n < NT; n += 2)
      if (n < nt) {
        uint32_t b[4];
        gm_ldsm_t(b, pb + 16 * n);
        float p[2][4];
        gm_mma16_0(p[0], o, b[0], b[1]);
        gm_mma16_0(p[1], o, b[2], b[3]);
        gm_mma16(p[0], h, b[0], b[1]);
        gm_mma16(p[1], h, b[2], b[3]);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[n + m][e] = fmaf(p[m][e], e < 2 ? sc.x : sc.y, acc[n + m][e]);
      }
  }
}
// A rows i0.. of a matrix with a factor for each row; (TRANS: columns i0..) of one with a factor a block
template <int NT>
__device__ __forceinline__ void gs_product_rows(float (&acc)[NT][4], int nt, int l0, int l1, const GsByRow& A, int i0, GmTile y, int j0) {
  const int lane = threadIdx.x & 31;
  const float* f = A.inv_s + (i0 + (lane >> 2)) * A.fr + (l0 >> 4) * A.fc;
  gs_product<NT, false>(acc, nt, l0, l1, A.hi, A.lo, i0 * A.pitch + gm_off_a(lane, A.pitch) + l0, 32u, y, j0, [&] {
    const float2 r = make_float2(f[0], f[8 * A.fr]);
    f += A.fc;
    return r;
  });
}
template <int NT, bool TRANS>
__device__ __forceinline__ void gs_product_a(float (&acc)[NT][4], int nt, int l0, int l1, const GsSplit& A, int i0, GmTile y, int j0) {
  const int lane = threadIdx.x & 31;
  const float* f = A.inv_s + (TRANS ? (i0 >> 4) + (l0 >> 4) * A.sp : (i0 >> 4) * A.sp + (l0 >> 4));
  gs_product<NT, TRANS>(acc, nt, l0, l1, A.hi, A.lo, TRANS ? i0 + gm_off_b(lane, A.pitch) + l0 * A.pitch : i0 * A.pitch + gm_off_a(lane, A.pitch) + l0,
                        TRANS ? 32u * A.pitch : 32u, y, j0, [&] {
                          const float r = *f;
                          f += TRANS ? A.sp : 1;
                          return make_float2(r, r);
                        });
}
// the same with A rows i0.. of an fp16 tile stored along l and B the split matrix, stored along j (ALONG_J) or along l
template <int NT, bool ALONG_J>
__device__ __forceinline__ void gs_product_b(float (&acc)[NT][4], int nt, int l1, GmTile x, int i0, const GsSplit& B, int j0) {
  const int lane = threadIdx.x & 31;
  uint32_t pa = gm_addr(x.p + i0 * x.pitch + gm_off_a(lane, x.pitch));
  uint32_t ph = gm_addr(B.hi + (ALONG_J ? j0 + gm_off_a(lane, B.pitch) : j0 * B.pitch + gm_off_b(lane, B.pitch)));
  const uint32_t lo = (uint32_t)((const char*)B.lo - (const char*)B.hi), dl = ALONG_J ? 32u * B.pitch : 32u, dn = ALONG_J ? 16u : 16u * B.pitch;
  const float* f = B.inv_s + (ALONG_J ? j0 >> 4 : (j0 >> 4) * B.sp);
  const int fl = ALONG_J ? B.sp : 1, fn = ALONG_J ? 1 : B.sp;
#pragma unroll 1
  for (int l = 0; l < l1; l += 16, pa += 32, ph += dl, f += fl) {
    uint32_t a[4];
    gm_ldsm(a, pa);
#pragma unroll
    for (int n = 0; n < NT; n += 2)
      if (n < nt) {
        uint32_t h[4], o[4];
        if (ALONG_J) { gm_ldsm_t(h, ph + n * dn); gm_ldsm_t(o, ph + n * dn + lo); }
        else { gm_ldsm(h, ph + n * dn); gm_ldsm(o, ph + n * dn + lo); }
        const float sc = f[(n >> 1) * fn];
        float p[2][4];
        gm_mma16_0(p[0], a, o[0], o[1]);
        gm_mma16_0(p[1], a, o[2], o[3]);
        gm_mma16(p[0], a, h[0], h[1]);
        gm_mma16(p[1], a, h[2], h[3]);
        gs_add(acc[n], p[0], sc);
        gs_add(acc[n + 1], p[1], sc);
      }
  }
}

// w / n and w % n of a warp's work items (w n < 2^18) without the division's thirty instructions
struct GsDiv {
  int n;
  uint32_t inv;
  __device__ __forceinline__ explicit GsDiv(int n_) : n(n_), inv((1u << 18) / (uint32_t)n_ + 1u) {}
  __device__ __forceinline__ void operator()(int w, int& q, int& r) const {
    q = (int)((uint32_t)w * inv >> 18);
    r = w - q * n;
  }
};

// ---- shared steps ----------------------------------------------------------------------------------------------------------------
// the state in fp32 and, SPLIT, as operand (zeros in the pad rows and columns), a warp per block
template <bool SPLIT>
__device__ __forceinline__ void gs_state_in(float* S, float* z, const GsLayout& L, const GsSplit& op, const float* s_in, const float* z_in, int K, int d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, nb = L.dp / 16;
  const GsDiv by(nb);
  for (int w = warp; w < (L.Kp / 16) * nb; w += blockDim.x >> 5) {
    int i0, j0;
    by(w, i0, j0);
    i0 *= 16; j0 *= 16;
    float a[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + g + 8 * r, j = j0 + 8 * n + 2 * t;
        const float2 v = s_in && i < K && j < d ? *reinterpret_cast<const float2*>(s_in + (size_t)i * d + j) : make_float2(0.f, 0.f);
        a[n][2 * r] = v.x; a[n][2 * r + 1] = v.y;
        if (j < d) *reinterpret_cast<float2*>(S + i * L.ps + j) = v;
      }
    if (SPLIT) gs_put(op, i0, j0, a);
  }
  for (int i = threadIdx.x; i < L.Kp; i += blockDim.x) z[i] = z_in && i < K ? z_in[i] : 0.f;
}
__device__ __forceinline__ void gs_state_out(const float* S, const float* z, const GsLayout& L, float* s_out, float* z_out, int K, int d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, nb = L.dp / 16;
  const GsDiv by(nb);
  for (int w = warp; w < (L.Kp / 16) * nb; w += blockDim.x >> 5) {
    int i0, j0;
    by(w, i0, j0);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 * 16 + g + 8 * (e >> 1), j = j0 * 16 + 8 * (e & 1) + 2 * t;
      if (i < K && j < d) *reinterpret_cast<float2*>(s_out + (size_t)i * d + j) = *reinterpret_cast<const float2*>(S + i * L.ps + j);
    }
  }
  for (int i = threadIdx.x; i < K; i += blockDim.x) z_out[i] = z[i];
}
// inv, gz and gz in two fp16 parts (a factor per 16 tokens) of a chunk's rows, from what sweep 1 left
struct GsRows {
  float *inv, *gz;
  __half *z_hi, *z_lo;
  float* z_f;
};
__device__ __forceinline__ GsRows gs_rows_at(float* row, int C) { return GsRows{row, row + C, (__half*)(row + 2 * C), (__half*)(row + 2 * C) + C, row + 3 * C}; }
__device__ __forceinline__ void gs_row_scalars(const GsRows& r, const float* ws_den, const float* ws_gz, int C, size_t base, int valid) {
  const int i = threadIdx.x;
  if (i >= ((C + 31) & ~31)) return;                 // whole warps
  const bool live = i < valid;                       // valid <= C
  const float inv = live ? 1.f / fmaxf(ws_den[base + i], kEps) : 0.f, gz = live ? ws_gz[base + i] : 0.f;
  uint32_t mag = gs_mag(gz) < kGsInf ? gs_mag(gz) : 0u;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, o));
  float s, inv_s;
  gs_factors(mag, s, inv_s);
  uint32_t hi, lo;
  gs_parts<true>(gz, 0.f, s, hi, lo);
  if (i < C) {
    r.inv[i] = inv; r.gz[i] = gz;
    reinterpret_cast<uint16_t*>(r.z_hi)[i] = (uint16_t)hi;
    reinterpret_cast<uint16_t*>(r.z_lo)[i] = (uint16_t)lo;
    if ((i & 15) == 0) r.z_f[i >> 4] = inv_s;
  }
}
// inv g as operand, blocks of 16 x 16 from item `w0` on in steps of `dw`; a factor for each column of a block, which is one column of the fp32 state
// that it is summed into.  The factors are powers of two, whose lower 16 bits are zero: a word holds two columns' (floats would take (128, 96) its
// chunks of 64)
__device__ __forceinline__ uint32_t* gs_col_factors(const GsSplit& G, int i0, int j) { return reinterpret_cast<uint32_t*>(G.inv_s) + ((i0 >> 4) * G.sp + j) / 2; }
template <int C>
__device__ __forceinline__ void gs_scale_rows(const GsSplit& G, GmTile y, const float* inv, int d, int w0, int dw) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, nb = G.sp / 16;
  const GsDiv by(nb);
  for (int w = w0; w < (C / 16) * nb; w += dw) {
    int i0, j0;
    by(w, i0, j0);
    i0 *= 16; j0 *= 16;
    float a[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + g + 8 * r, j = j0 + 8 * n + 2 * t;
        const float2 v = j < d ? gm_row(y, i, j) : make_float2(0.f, 0.f);
        a[n][2 * r] = v.x * inv[i]; a[n][2 * r + 1] = v.y * inv[i];
      }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      float f[2], inv_f[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t x = gs_mag(a[n][e]), y = gs_mag(a[n][2 + e]);
        uint32_t mag = max(x < kGsInf ? x : 0u, y < kGsInf ? y : 0u);
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, o));
        gs_factors(mag, f[e], inv_f[e]);
      }
      const int j = j0 + 8 * n + 2 * t;
      if (g == 0) *gs_col_factors(G, i0, j) = __float_as_uint(inv_f[0]) >> 16 | __float_as_uint(inv_f[1]);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t hi, lo;
        gs_parts<true>(a[n][2 * r] * f[0], a[n][2 * r + 1] * f[1], 1.f, hi, lo);
        *reinterpret_cast<uint32_t*>(G.hi + (i0 + g + 8 * r) * G.pitch + j) = hi;
        *reinterpret_cast<uint32_t*>(G.lo + (i0 + g + 8 * r) * G.pitch + j) = lo;
      }
    }
  }
}
__device__ __forceinline__ uint32_t gs_pair(const __half* p) { return *reinterpret_cast<const uint32_t*>(p); }
// S += X^T Y, z += colsum(X) over a chunk -- WEIGHTED: X^T G with G the split inv g, and X^T gz -- summed in registers from zero, then added
// to the fp32 state with one rounding; SPLIT: the new block as operand.  A warp per block of S; those of its first columns take z.
template <int C, bool WEIGHTED, bool SPLIT>
__device__ __forceinline__ void gs_update(float* S, float* z, const GsLayout& L, const GsSplit& op, GmTile x, GmTile y, const GsSplit& G, const GsRows& rows,
                                          int K, int d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, nb = L.dp / 16;
  const GsDiv by(nb);
  for (int w = warp; w < (L.Kp / 16) * nb; w += blockDim.x >> 5) {
    int i0, j0;
    by(w, i0, j0);
    i0 *= 16; j0 *= 16;
    float acc[2][4], az[4] = {};
    gm_zero(acc);
    const uint32_t pa = gm_addr(x.p + i0 + gm_off_b(lane, x.pitch)), da = 2u * x.pitch;
    const uint32_t pb = gm_addr(WEIGHTED ? G.hi + j0 + gm_off_a(lane, G.pitch) : y.p + j0 + gm_off_a(lane, y.pitch)), db = 2u * (WEIGHTED ? G.pitch : y.pitch);
    const uint32_t lo = WEIGHTED ? (uint32_t)((const char*)G.lo - (const char*)G.hi) : 0u;
#pragma unroll
    for (int l = 0; l < C; l += 16) {
      uint32_t a[4], b[4], o[4];
      float p[2][4];
      gm_ldsm_t(a, pa + l * da);
      if (WEIGHTED) {
        gm_ldsm_t(b, pb + l * db);
        gm_ldsm_t(o, pb + l * db + lo);
        gm_mma16_0(p[0], a, o[0], o[1]);
        gm_mma16_0(p[1], a, o[2], o[3]);
        gm_mma16(p[0], a, b[0], b[1]);
        gm_mma16(p[1], a, b[2], b[3]);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const uint32_t sc = *gs_col_factors(G, l, j0 + 8 * n + 2 * t);
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[n][e] = fmaf(p[n][e], __uint_as_float(e & 1 ? sc & 0xFFFF0000u : sc << 16), acc[n][e]);
        }
        if (j0 == 0) {
          const uint32_t h0 = g == 0 ? gs_pair(rows.z_hi + l + 2 * t) : 0u, h1 = g == 0 ? gs_pair(rows.z_hi + l + 8 + 2 * t) : 0u;
          const uint32_t o0 = g == 0 ? gs_pair(rows.z_lo + l + 2 * t) : 0u, o1 = g == 0 ? gs_pair(rows.z_lo + l + 8 + 2 * t) : 0u;
          float q[4];
          gm_mma16_0(q, a, o0, o1);
          gm_mma16(q, a, h0, h1);
          gs_add(az, q, rows.z_f[l >> 4]);
        }
      } else {
        gm_ldsm_t(b, pb + l * db);
        gm_mma16_0(p[0], a, b[0], b[1]);
        gm_mma16_0(p[1], a, b[2], b[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) { acc[0][e] += p[0][e]; acc[1][e] += p[1][e]; }
        if (j0 == 0) {
          const uint32_t ones = g == 0 ? 0x3C003C00u : 0u;
          float q[4];
          gm_mma16_0(q, a, ones, ones);
#pragma unroll
          for (int e = 0; e < 4; ++e) az[e] += q[e];
        }
      }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + g + 8 * r, j = j0 + 8 * n + 2 * t;
        float2 v = make_float2(0.f, 0.f);
        if (j < d) {
          float2* p = reinterpret_cast<float2*>(S + i * L.ps + j);
          v = *p;
          v.x += acc[n][2 * r]; v.y += acc[n][2 * r + 1];
          *p = v;
        }
        acc[n][2 * r] = i < K ? v.x : 0.f; acc[n][2 * r + 1] = i < K ? v.y : 0.f;      // the operand's pad rows meet pad columns of X tiles
      }
    if (SPLIT) gs_put(op, i0, j0, acc);
    if (j0 == 0 && t == 0) { z[i0 + g] += az[0]; z[i0 + g + 8] += az[2]; }
  }
}
// the w-th 16 x 16 block on or below the diagonal
__device__ __forceinline__ void gs_lower(int w, int& mi, int& ni) {
  mi = w >= 6 ? 3 : w >= 3 ? 2 : w >= 1 ? 1 : 0;
  ni = w - mi * (mi + 1) / 2;
}

// ===========================================================================================================================
// forward.  grid (BH, nseg); s_seg / z_seg: the state entering each segment (null = zero)
// ===========================================================================================================================
template <int C>
__global__ void __maxnreg__(kGsRegs)
gs_causal_fwd_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, __half* __restrict__ out,
                     const float* __restrict__ s_seg, const float* __restrict__ z_seg, float* __restrict__ s_out, float* __restrict__ z_out,
                     float* __restrict__ den_out, int64_t T, int BH, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gs_raw[];
  const GsLayout L = gs_layout_fwd(C, K, d);
  constexpr int MT = C / 16;
  float *S = (float*)(gs_raw + L.S), *z = (float*)(gs_raw + L.z), *rs = (float*)(gs_raw + L.row), *qz = rs + MT * C;
  const GsSplit op = gs_split_at(gs_raw, L.s_hi, L.s_f, L.Kp, L.ph, L.dp / 16);
  // a token's output is divided by its own denominator: weights of another in its block may be any times larger than its own
  const GsByRow P{(__half*)(gs_raw + L.P), (__half*)(gs_raw + L.P) + C * L.pc, (float*)(gs_raw + L.p_f), L.pc, 1, C};
  const int bh = blockIdx.x, seg = blockIdx.y, nseg = gridDim.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = (int)((t_end - t_begin + C - 1) / C);
  const size_t slot = (size_t)bh * nseg + seg;
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto tile = [&](int which) {              // 0 q, 1 k, 2 v
    return GmTile{(const __half*)(gs_raw + L.tile + which * L.x_bytes), which < 2 ? L.px : L.py};
  };
  const int ng = L.dp / 16;
  const GsDiv by_ng(ng);
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {
    if (c < nchunk) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(0).p, L.px, q, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(1).p, L.px, k, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(2).p, L.py, v, C, d, walk_y, t0, valid, BH, bh, nullptr);
    }
    gm_commit();
  };
  for (int i = 0; i < 3; ++i) gm_pad(tile(i), C, i < 2 ? K : d);
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(0);
  gs_state_in<true>(S, z, L, op, s_seg ? s_seg + slot * K * d : nullptr, z_seg ? z_seg + slot * K : nullptr, K, d);
  for (int c = 0; c < nchunk; ++c) {
    if (c == nchunk - 1 && gs_pdl(tseg, C)) sm100::pdl_launch_dependents();
    gm_wait<0>();
    const GmTile tq = tile(0), tk = tile(1), tv = tile(2);
    const int64_t t0 = t_begin + (int64_t)c * C;
    const int valid = (int)min((int64_t)C, t_end - t0);
    const bool odd = __syncthreads_or(gm_odd(tv.p, tv.pitch, C, walk_y)) != 0;      // the tiles have landed, the state is new
    // P = tril(Q K^T), its row sums per 16 columns, q . z
    for (int w = warp; w < MT * (MT + 1) / 2; w += nw) {
      int mi, ni;
      gs_lower(w, mi, ni);
      const int i0 = mi * 16, j0 = ni * 16;
      float acc[2][4];
      gm_zero(acc);
      gm_exact(acc, tq, i0, tk, j0, K);
      float r[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (j0 + 8 * n + 2 * t + (e & 1) > i0 + g + 8 * (e >> 1)) acc[n][e] = 0.f;
          r[e >> 1] += acc[n][e];
        }
      gs_put_rows(P, i0, j0, acc);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        r[e] = gm_quad(r[e]);
        if (t == 0) rs[ni * C + i0 + g + 8 * e] = r[e];
      }
    }
    gm_qz<C>(qz, tq, z, K);
    __syncthreads();
    // out = (P V + Q S) / max(raw, 1)
    for (int w = warp; w < MT * ng; w += nw) {
      int mi, ni;
      by_ng(w, mi, ni);
      const int i0 = mi * 16, j0 = ni * 16, nt = min(2, (d - j0) / 8);
      float acc[2][4];
      gm_zero(acc);
      if (odd) gm_product_masked<2>(acc, i0, j0, nt, 0, i0 + 16, [=](int i, int l) { return make_float2(gs_at(P, i, l), gs_at(P, i, l + 1)); },
                                    [=](int l, int j) { return gm_col(tv, l, j); }, [](int i, int l) { return l <= i; });
      else gs_product_rows<2>(acc, nt, 0, i0 + 16, P, i0, tv, j0);
      gs_product_b<2, true>(acc, nt, K, tq, i0, op, j0);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + g + 8 * r;
        float raw = qz[i];
        for (int b = 0; b <= mi; ++b) raw += rs[b * C + i];
        if (i >= valid) continue;
        const size_t row = (size_t)(t0 + i) * BH + bh;
        const float inv = 1.f / fmaxf(raw, kEps);
        if (den_out && j0 == 0 && t == 0) den_out[(size_t)bh * T + t0 + i] = raw;
#pragma unroll
        for (int n = 0; n < 2; ++n)
          if (n < nt) gm_store2(out + row * d + j0 + 8 * n + 2 * t, acc[n][2 * r] * inv, acc[n][2 * r + 1] * inv);
      }
    }
    __syncthreads();
    if (c + 1 < nchunk || s_out) gs_update<C, false, true>(S, z, L, op, tk, tv, op, GsRows{}, K, d);
    __syncthreads();
    load(c + 1);
  }
  if (s_out && seg == nseg - 1) {
    __syncthreads();
    gs_state_out(S, z, L, s_out + (size_t)bh * K * d, z_out + (size_t)bh * K, K, d);
  }
}

// ===========================================================================================================================
// backward, sweep 1: gq, raw denominators, gz
// ===========================================================================================================================
template <int C>
__global__ void __maxnreg__(kGsRegs)
gs_causal_bwd_q_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, const __half* __restrict__ gr,
                       __half* __restrict__ gq, const float* __restrict__ s_seg, const float* __restrict__ z_seg,
                       float* __restrict__ ws_den, float* __restrict__ ws_gz, int64_t T, int BH, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gs_raw[];
  const GsLayout L = gs_layout_q(C, K, d);
  constexpr int MT = C / 16, kTri = MT * (MT + 1) / 2, kHold = (kTri + 7) / 8;      // blocks a warp of eight or more holds at most
  const int kg = gm_groups32(K);
  float *S = (float*)(gs_raw + L.S), *z = (float*)(gs_raw + L.z), *rs = (float*)(gs_raw + L.row), *pg = rs + MT * C, *wq = pg + MT * C,
        *qz = wq + kg * C, *inv = qz + C, *gz = inv + C;
  const GsSplit op = gs_split_at(gs_raw, L.s_hi, L.s_f, L.Kp, L.ph, L.dp / 16), D = gs_split_at(gs_raw, L.D, L.d_f, C, L.pc, MT);
  const int bh = blockIdx.x, seg = blockIdx.y, nseg = gridDim.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = (int)((t_end - t_begin + C - 1) / C);
  const size_t slot = (size_t)bh * nseg + seg;
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto tile = [&](int which) {              // 0 q, 1 k, 2 v, 3 g
    return GmTile{(const __half*)(gs_raw + L.tile + (which < 2 ? which * L.x_bytes : 2 * L.x_bytes + (which - 2) * L.y_bytes)), which < 2 ? L.px : L.py};
  };
  const GsDiv by_kg(kg);
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {
    if (c < nchunk) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(0).p, L.px, q, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(1).p, L.px, k, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(2).p, L.py, v, C, d, walk_y, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(3).p, L.py, gr, C, d, walk_y, t0, valid, BH, bh, nullptr);
    }
    gm_commit();
  };
  for (int i = 0; i < 4; ++i) gm_pad(tile(i), C, i < 2 ? K : d);
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(0);
  gs_state_in<true>(S, z, L, op, s_seg ? s_seg + slot * K * d : nullptr, z_seg ? z_seg + slot * K : nullptr, K, d);
  for (int c = 0; c < nchunk; ++c) {
    if (c == nchunk - 1 && gs_pdl(tseg, C)) sm100::pdl_launch_dependents();
    gm_wait<0>();
    const GmTile tq = tile(0), tk = tile(1), tv = tile(2), tg = tile(3);
    const int64_t t0 = t_begin + (int64_t)c * C;
    const int valid = (int)min((int64_t)C, t_end - t0);
    const bool odd = __syncthreads_or(gm_odd(tk.p, tk.pitch, C, walk_x)) != 0;
    // G = g V^T on and below the diagonal, held; per 16 columns the row sums of P and of P o G
    float G[kHold][2][4];
#pragma unroll
    for (int u = 0; u < kHold; ++u) {
      const int w = warp + u * nw;
      if (w >= kTri) continue;
      int mi, ni;
      gs_lower(w, mi, ni);
      const int i0 = mi * 16, j0 = ni * 16;
      float p[2][4];
      gm_zero(p); gm_zero(G[u]);
      gm_exact(p, tq, i0, tk, j0, K);
      gm_exact(G[u], tg, i0, tv, j0, d);
      float r[2] = {0.f, 0.f}, s[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (j0 + 8 * n + 2 * t + (e & 1) <= i0 + g + 8 * (e >> 1)) { r[e >> 1] += p[n][e]; s[e >> 1] = fmaf(p[n][e], G[u][n][e], s[e >> 1]); }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        r[e] = gm_quad(r[e]); s[e] = gm_quad(s[e]);
        if (t == 0) { rs[ni * C + i0 + g + 8 * e] = r[e]; pg[ni * C + i0 + g + 8 * e] = s[e]; }
      }
    }
    // W = g S^T: the row sums of Q o W per 32 features (from the last warp on: the first ones have two blocks above)
    for (int w = nw - 1 - warp; w < MT * kg; w += nw) {
      int mi, gi;
      by_kg(w, mi, gi);
      const int i0 = mi * 16, j0 = gi * 32, nt = min(4, (K - j0) / 8);
      float a[4][4];
      gm_zero(a);
      gs_product_b<4, false>(a, nt, d, tg, i0, op, j0);
      float s[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < 4; ++n)
        if (n < nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float2 x = gm_row(tq, i0 + g + 8 * e, j0 + 8 * n + 2 * t);
            s[e] = fmaf(x.x, a[n][2 * e], fmaf(x.y, a[n][2 * e + 1], s[e]));
          }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        s[e] = gm_quad(s[e]);
        if (t == 0) wq[gi * C + i0 + g + 8 * e] = s[e];
      }
    }
    gm_qz<C>(qz, tq, z, K);
    __syncthreads();
    // inv and gz of each row; D = tril(inv G + gz)
    auto scalars = [&](int i, float& iv, float& gzv) {
      float raw = qz[i], gn = 0.f;
      for (int b = 0; b <= i / 16; ++b) { raw += rs[b * C + i]; gn += pg[b * C + i]; }
      for (int b = 0; b < kg; ++b) gn += wq[b * C + i];
      iv = 1.f / fmaxf(raw, kEps);
      gzv = raw > kEps ? -gn * iv * iv : 0.f;                      // strict >, upstream rfa.py:91
      return raw;
    };
    if (threadIdx.x < C) {
      const int i = threadIdx.x;
      float iv, gzv;
      const float raw = scalars(i, iv, gzv);
      inv[i] = iv; gz[i] = gzv;
      if (i < valid) { ws_den[(size_t)bh * T + t0 + i] = raw; ws_gz[(size_t)bh * T + t0 + i] = gzv; }
    }
#pragma unroll
    for (int u = 0; u < kHold; ++u) {
      const int w = warp + u * nw;
      if (w >= kTri) continue;
      int mi, ni;
      gs_lower(w, mi, ni);
      const int i0 = mi * 16, j0 = ni * 16;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float iv, gzv;
        scalars(i0 + g + 8 * r, iv, gzv);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            G[u][n][2 * r + e] = j0 + 8 * n + 2 * t + e <= i0 + g + 8 * r ? fmaf(iv, G[u][n][2 * r + e], gzv) : 0.f;
      }
      gs_put(D, i0, j0, G[u]);
    }
    __syncthreads();
    // gq = inv W + D K + gz z
    for (int w = warp; w < MT * kg; w += nw) {
      int mi, gi;
      by_kg(w, mi, gi);
      const int i0 = mi * 16, j0 = gi * 32, nt = min(4, (K - j0) / 8);
      float a[4][4];
      gm_zero(a);
      gs_product_b<4, false>(a, nt, d, tg, i0, op, j0);
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[n][e] *= inv[i0 + g + 8 * (e >> 1)];
      if (odd) gm_product_masked<4>(a, i0, j0, nt, 0, i0 + 16, [=](int i, int l) { return make_float2(gs_at(D, i, l), gs_at(D, i, l + 1)); },
                                    [=](int l, int j) { return gm_col(tk, l, j); }, [](int i, int l) { return l <= i; });
      else gs_product_a<4, false>(a, nt, 0, i0 + 16, D, i0, tk, j0);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = i0 + g + 8 * r;
        if (i >= valid) continue;
        __half* dst = gq + ((size_t)(t0 + i) * BH + bh) * K;
#pragma unroll
        for (int n = 0; n < 4; ++n)
          if (n < nt) {
            const int j = j0 + 8 * n + 2 * t;
            gm_store2(dst + j, fmaf(gz[i], z[j], a[n][2 * r]), fmaf(gz[i], z[j + 1], a[n][2 * r + 1]));
          }
      }
    }
    __syncthreads();
    if (c + 1 < nchunk) gs_update<C, false, true>(S, z, L, op, tk, tv, op, GsRows{}, K, d);
    __syncthreads();
    load(c + 1);
  }
}

// ===========================================================================================================================
// backward, sweep 2 (chunks in reverse): gk, gv
// ===========================================================================================================================
template <int C>
__global__ void __maxnreg__(kGsRegs)
gs_causal_bwd_kv_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, const __half* __restrict__ gr,
                        __half* __restrict__ gk, __half* __restrict__ gv, const float* __restrict__ ws_den, const float* __restrict__ ws_gz,
                        const float* __restrict__ ds_seg, const float* __restrict__ dz_seg, int64_t T, int BH, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gs_raw[];
  const GsLayout L = gs_layout_kv(C, K, d);
  constexpr int MT = C / 16, kTri = MT * (MT + 1) / 2;
  const int kg = gm_groups32(K);
  float *S = (float*)(gs_raw + L.S), *z = (float*)(gs_raw + L.z);
  const GsRows rows = gs_rows_at((float*)(gs_raw + L.row), C);
  const GsSplit op = gs_split_at(gs_raw, L.s_hi, L.s_f, L.Kp, L.ph, L.dp / 16), P = gs_split_at(gs_raw, L.P, L.p_f, C, L.pc, MT),
                D = gs_split_at(gs_raw, L.D, L.d_f, C, L.pc, MT), Gs = gs_split_at(gs_raw, L.G, L.g_f, C, L.ph, L.dp);
  const int bh = blockIdx.x, seg = blockIdx.y, nseg = gridDim.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = (int)((t_end - t_begin + C - 1) / C);
  const size_t slot = (size_t)bh * nseg + seg;
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  auto tile = [&](int which) {              // 0 q, 1 k, 2 v, 3 g
    return GmTile{(const __half*)(gs_raw + L.tile + (which < 2 ? which * L.x_bytes : 2 * L.x_bytes + (which - 2) * L.y_bytes)), which < 2 ? L.px : L.py};
  };
  const int ng = L.dp / 16;
  const GsDiv by_kg(kg), by_ng(ng);
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {      // c counts down to 0
    if (c >= 0) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(0).p, L.px, q, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(1).p, L.px, k, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(2).p, L.py, v, C, d, walk_y, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(3).p, L.py, gr, C, d, walk_y, t0, valid, BH, bh, nullptr);
    }
    gm_commit();
  };
  for (int i = 0; i < 4; ++i) gm_pad(tile(i), C, i < 2 ? K : d);
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(nchunk - 1);
  gs_state_in<true>(S, z, L, op, ds_seg ? ds_seg + slot * K * d : nullptr, dz_seg ? dz_seg + slot * K : nullptr, K, d);
  for (int c = nchunk - 1; c >= 0; --c) {
    if (c == 0 && gs_pdl(tseg, C)) sm100::pdl_launch_dependents();
    const int64_t t0 = t_begin + (int64_t)c * C;
    const int valid = (int)min((int64_t)C, t_end - t0);
    gs_row_scalars(rows, ws_den, ws_gz, C, (size_t)bh * T + t0, valid);
    gm_wait<0>();
    const GmTile tq = tile(0), tk = tile(1), tv = tile(2), tg = tile(3);
    const bool odd = __syncthreads_or(gm_odd(tq.p, tq.pitch, C, walk_x) || gm_odd(tg.p, tg.pitch, C, walk_y)) != 0;
    // P' = inv tril(Q K^T), D = tril(inv g V^T + gz), inv g
    for (int w = warp; w < kTri; w += nw) {
      int mi, ni;
      gs_lower(w, mi, ni);
      const int i0 = mi * 16, j0 = ni * 16;
      float p[2][4], a[2][4];
      gm_zero(p); gm_zero(a);
      gm_exact(p, tq, i0, tk, j0, K);
      gm_exact(a, tg, i0, tv, j0, d);
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = j0 + 8 * n + 2 * t + (e & 1), i = i0 + g + 8 * (e >> 1);
          p[n][e] = j <= i ? p[n][e] * rows.inv[i] : 0.f;
          a[n][e] = j <= i ? fmaf(a[n][e], rows.inv[i], rows.gz[i]) : 0.f;
        }
      gs_put(P, i0, j0, p);
      gs_put(D, i0, j0, a);
    }
    if (c > 0) gs_scale_rows<C>(Gs, tg, rows.inv, d, nw - 1 - warp, nw);
    __syncthreads();
    // gk = D^T Q + V dS^T + dz   and   gv = P'^T g + K dS
    for (int w = warp; w < MT * (kg + ng); w += nw) {
      if (w < MT * kg) {
        int mi, gi;
        by_kg(w, mi, gi);
        const int i0 = mi * 16, j0 = gi * 32, nt = min(4, (K - j0) / 8);
        float a[4][4];
        gm_zero(a);
        if (odd) gm_product_masked<4>(a, i0, j0, nt, i0, C, [=](int i, int l) { return make_float2(gs_at(D, l, i), gs_at(D, l + 1, i)); },
                                      [=](int l, int j) { return gm_col(tq, l, j); }, [](int i, int l) { return l >= i; });
        else gs_product_a<4, true>(a, nt, i0, C, D, i0, tq, j0);
        gs_product_b<4, false>(a, nt, d, tv, i0, op, j0);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int i = i0 + g + 8 * r;
          if (i >= valid) continue;
          __half* dst = gk + ((size_t)(t0 + i) * BH + bh) * K;
#pragma unroll
          for (int n = 0; n < 4; ++n)
            if (n < nt) {
              const int j = j0 + 8 * n + 2 * t;
              gm_store2(dst + j, a[n][2 * r] + z[j], a[n][2 * r + 1] + z[j + 1]);
            }
        }
      } else {
        int mi, ni;
        by_ng(w - MT * kg, mi, ni);
        const int i0 = mi * 16, j0 = ni * 16, nt = min(2, (d - j0) / 8);
        float a[2][4];
        gm_zero(a);
        if (odd) gm_product_masked<2>(a, i0, j0, nt, i0, C, [=](int i, int l) { return make_float2(gs_at(P, l, i), gs_at(P, l + 1, i)); },
                                      [=](int l, int j) { return gm_col(tg, l, j); }, [](int i, int l) { return l >= i; });
        else gs_product_a<2, true>(a, nt, i0, C, P, i0, tg, j0);
        gs_product_b<2, true>(a, nt, K, tk, i0, op, j0);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int i = i0 + g + 8 * r;
          if (i >= valid) continue;
          __half* dst = gv + ((size_t)(t0 + i) * BH + bh) * d;
#pragma unroll
          for (int n = 0; n < 2; ++n)
            if (n < nt) gm_store2(dst + j0 + 8 * n + 2 * t, a[n][2 * r], a[n][2 * r + 1]);
        }
      }
    }
    __syncthreads();
    if (c > 0) gs_update<C, true, true>(S, z, L, op, tq, tg, Gs, rows, K, d);
    __syncthreads();
    load(c - 1);
  }
}

// ===========================================================================================================================
// state reduction over runs of tokens: sum x (x) y, sum x (padded keys left out), or with ws_den / ws_gz the reverse one,
// sum x (x) (inv y), sum gz x.  grid (BH, runs <= nseg)
// ===========================================================================================================================
template <int C, bool WEIGHTED>
__global__ void __maxnreg__(kGsRegs)
gs_state_kernel(const __half* __restrict__ x, const __half* __restrict__ y, const uint8_t* __restrict__ pad_mask,
                const float* __restrict__ ws_den, const float* __restrict__ ws_gz, float* __restrict__ s_out, float* __restrict__ z_out,
                int64_t T, int BH, int H, int nseg, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gs_raw[];
  const GsLayout L = gs_layout_state(C, K, d, WEIGHTED);
  float *S = (float*)(gs_raw + L.S), *z = (float*)(gs_raw + L.z);
  const GsRows rows = gs_rows_at((float*)(gs_raw + L.row), C);
  const GsSplit Gs = gs_split_at(gs_raw, L.G, L.g_f, C, L.ph, L.dp);
  const int bh = blockIdx.x, seg = blockIdx.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = t_end > t_begin ? (int)((t_end - t_begin + C - 1) / C) : 0;
  const size_t slot = (size_t)bh * nseg + seg;
  const uint8_t* mrow = pad_mask ? pad_mask + (size_t)(bh / H) * T : nullptr;
  auto tile = [&](int which) { return GmTile{(const __half*)(gs_raw + L.tile + which * L.x_bytes), which < 1 ? L.px : L.py}; };
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {
    if (c < nchunk) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(0).p, L.px, x, C, K, walk_x, t0, valid, BH, bh, mrow);
      gm_load((__half*)tile(1).p, L.py, y, C, d, walk_y, t0, valid, BH, bh, mrow);
    }
    gm_commit();
  };
  for (int i = 0; i < 2; ++i) gm_pad(tile(i), C, i < 1 ? K : d);
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(0);
  gs_state_in<false>(S, z, L, Gs, nullptr, nullptr, K, d);
  for (int c = 0; c < nchunk; ++c) {
    if (c == nchunk - 1 && gs_pdl(tseg, C)) sm100::pdl_launch_dependents();
    const int64_t t0 = t_begin + (int64_t)c * C;
    if (WEIGHTED) gs_row_scalars(rows, ws_den, ws_gz, C, (size_t)bh * T + t0, (int)min((int64_t)C, t_end - t0));
    gm_wait<0>();
    __syncthreads();
    if (WEIGHTED) {
      gs_scale_rows<C>(Gs, tile(1), rows.inv, d, threadIdx.x >> 5, blockDim.x >> 5);
      __syncthreads();
    }
    gs_update<C, WEIGHTED, false>(S, z, L, Gs, tile(0), tile(1), Gs, rows, K, d);
    __syncthreads();
    load(c + 1);
  }
  __syncthreads();
  gs_state_out(S, z, L, s_out + slot * K * d, z_out + slot * K, K, d);
}

// ---------------------------------------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------------------------------------
constexpr uint32_t kGsSmemMax = 227 * 1024;
struct GsShape { int C, ctas, threads; };
// Which chunk.  A longer one shares the state's products, its update and the barriers among more tokens; shorter ones leave room for
// more CTAs on an SM, one of which works while another waits, and cut a sequence into more segments.  24 warps in all.
//
// Chunks of 64 wherever two of their CTAs fit an SM: us forward + backward, 64 / 32 / 16 tokens, (K, d) = (64, 32), 64 heads x 512 tokens 71 / 80 / 111,
// 128 x 1024 256 / 243 / 363, 64 x 45 21 / 27 / 27.  Where one fits, against those of 32 (of which one to three do), gs_cost decides; in units of an
// uncut chunk of 64 (23 to 40 us) it is a fit to 500 calls of 11 geometries, 0.4 % over the better of the two in the mean and 16 % at most:
// (64, 96), 148 heads x 1024 459 / 533, 96 x 1024 444 / 364, 64 x 512 144 / 145, 8 x 256 40 / 33, 64 x 45 28 / 42; (96, 96), 64 x 512 174 / 227 / 247,
// 128 x 1024 555 / 732 / 964; (64, 128) 175 / 227 / 239, 551 / 732 / 923.
// Chunks of 16 where two CTAs fit and only one of 32, and all of them at half of the SMs: (192, 48), 4 heads x 128 51 / 38 / 33, 16 x 128 52 / 39 / 46; and
// where nothing longer fits (there generic_mma.cu decides).
static float gs_cost(int C, int ctas, int64_t T, int BH, bool whole) {
  const CausalPlan p = cut_segments(T, C, whole ? 1 : kSms * ctas / BH, 1);
  const int64_t n = (int64_t)BH * p.nseg, fit = kSms * ctas, waves = (n + fit - 1) / fit, per_sm = (n + kSms - 1) / kSms;
  const float m = (float)(p.tseg / C);
  if (C == 64) return waves * (p.nseg == 1 ? m : 0.2f + 1.16f * m);      // a cut one makes the pre-pass too
  const float w = per_sm == 1 ? 0.75f : per_sm == 2 || ctas == 2 ? 1.1f : 1.42f;
  return waves * (p.nseg == 1 ? 0.82f * w * m : 0.35f + w * m);
}
// whole: the sequences are not cut (a call without a workspace, a state reduction alone)
static GsShape gs_shape(int64_t T, int BH, int K, int d, bool whole) {
  int ctas[3];                  // how many CTAs of chunks of 64, 32, 16 an SM holds
  for (int i = 0; i < 3; ++i) {
    const uint32_t a = gs_layout_q(64 >> i, K, d).total, b = gs_layout_kv(64 >> i, K, d).total, need = a > b ? a : b;
    const int n = (int)(kGsSmemMax / (need + 1024));
    ctas[i] = need > kGsSmemMax ? 0 : n < 1 ? 1 : n > 3 ? 3 : n;
  }
  int i = ctas[0] ? 0 : ctas[1] ? 1 : 2;
  if (ctas[0] == 1 && ctas[1] && gs_cost(32, ctas[1], T, BH, whole) < gs_cost(64, 1, T, BH, whole)) i = 1;
  if (ctas[0] < 2 && ctas[1] < 2 && ctas[2] > 1 && (T <= 16 || (!whole && (T + 15) / 16 * BH <= kSms / 2))) i = 2;
  return GsShape{ctas[i] ? 64 >> i : 0, ctas[i], ctas[i] == 3 ? 256 : ctas[i] == 2 ? 384 : 768};
}

// Tokens per chunk of these kernels, 0 when the geometry does not fit them; *ctas = how many of their CTAs one SM holds
int split_chunk(int64_t T, int BH, int K, int d, bool whole, int* ctas) {
  if (K <= 0 || d <= 0 || K % 8 || d % 8 || K > 1024 || d > 1024) return 0;
  const GsShape s = gs_shape(T, BH, K, d, whole);
  if (ctas) *ctas = s.ctas;
  return s.C;
}

template <class KERNEL, class... Args>
static int gs_launch(KERNEL kernel, const char* what, bool pdl, int threads, uint32_t smem, dim3 grid, cudaStream_t st, Args... args) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail((int)e, "%s: cannot reserve %u bytes of shared memory: %s", what, smem, cudaGetErrorString(e));
  if (pdl) sm100::launch_pdl(kernel, grid, dim3(threads), smem, st, args...);
  else kernel<<<grid, threads, smem, st>>>(args...);
  return check_launch(what);
}
#define RFA_GS_DISPATCH(shape, CALL)            \
  do {                                          \
    const GsShape gs_ = (shape);                \
    if (gs_.C == 64) { CALL(64); }              \
    if (gs_.C == 32) { CALL(32); }              \
    CALL(16);                                   \
  } while (0)

int launch_causal_split_fwd(const __half* q, const __half* k, const __half* v, __half* out, const float* s_seg, const float* z_seg, float* s_out,
                            float* z_out, float* den_out, int64_t T, int BH, int nseg, int64_t tseg, int K, int d, cudaStream_t st) {
#define RFA_GS_CALL(C) return gs_launch(gs_causal_fwd_kernel<C>, "rfa_causal_fwd (chunked)", gs_pdl(tseg, C), gs_.threads, gs_layout_fwd(C, K, d).total, \
                                        dim3(BH, nseg), st, q, k, v, out, s_seg, z_seg, s_out, z_out, den_out, T, BH, tseg, K, d)
  RFA_GS_DISPATCH(gs_shape(T, BH, K, d, nseg == 1), RFA_GS_CALL);
#undef RFA_GS_CALL
}
int launch_causal_split_bwd_q(const __half* q, const __half* k, const __half* v, const __half* g, __half* gq, const float* s_seg, const float* z_seg,
                              float* ws_den, float* ws_gz, int64_t T, int BH, int nseg, int64_t tseg, int K, int d, cudaStream_t st) {
#define RFA_GS_CALL(C) return gs_launch(gs_causal_bwd_q_kernel<C>, "rfa_causal_bwd_q (chunked)", gs_pdl(tseg, C), gs_.threads, gs_layout_q(C, K, d).total, \
                                        dim3(BH, nseg), st, q, k, v, g, gq, s_seg, z_seg, ws_den, ws_gz, T, BH, tseg, K, d)
  RFA_GS_DISPATCH(gs_shape(T, BH, K, d, nseg == 1), RFA_GS_CALL);
#undef RFA_GS_CALL
}
int launch_causal_split_bwd_kv(const __half* q, const __half* k, const __half* v, const __half* g, __half* gk, __half* gv, const float* ws_den,
                               const float* ws_gz, const float* ds_seg, const float* dz_seg, int64_t T, int BH, int nseg, int64_t tseg, int K,
                               int d, cudaStream_t st) {
#define RFA_GS_CALL(C) return gs_launch(gs_causal_bwd_kv_kernel<C>, "rfa_causal_bwd_kv (chunked)", gs_pdl(tseg, C), gs_.threads, gs_layout_kv(C, K, d).total, \
                                        dim3(BH, nseg), st, q, k, v, g, gk, gv, ws_den, ws_gz, ds_seg, dz_seg, T, BH, tseg, K, d)
  RFA_GS_DISPATCH(gs_shape(T, BH, K, d, nseg == 1), RFA_GS_CALL);
#undef RFA_GS_CALL
}
int launch_state_split(const __half* x, const __half* y, const uint8_t* pad_mask, const float* ws_den, const float* ws_gz, float* s, float* z,
                       int64_t T, int BH, int H, int nseg, int64_t tseg, int runs, int K, int d, cudaStream_t st) {
#define RFA_GS_CALL(C)                                                                                                                \
  return ws_den ? gs_launch(gs_state_kernel<C, true>, "state reduction (chunked)", gs_pdl(tseg, C), gs_.threads, gs_layout_state(C, K, d, true).total, \
                            dim3(BH, runs), st, x, y, pad_mask, ws_den, ws_gz, s, z, T, BH, H, nseg, tseg, K, d)                      \
                : gs_launch(gs_state_kernel<C, false>, "state reduction (chunked)", gs_pdl(tseg, C), gs_.threads, gs_layout_state(C, K, d, false).total, \
                            dim3(BH, runs), st, x, y, pad_mask, ws_den, ws_gz, s, z, T, BH, H, nseg, tseg, K, d)
  RFA_GS_DISPATCH(gs_shape(T, BH, K, d, nseg == 1), RFA_GS_CALL);
#undef RFA_GS_CALL
}

}  // namespace rfa
