// Causal RFA and the state reduction for geometries other than K = 128, d = 64, in chunks on the tensor cores.
//
// Any K % 8 == 0, d % 8 == 0 whose fp32 state and one chunk's tiles fit in shared memory (upstream takes any K % 16 == 0,
// d % 8 == 0, cuda/forward.cu:150-153); what does not fit stays on the token-at-a-time kernels of generic.cu, and those whose
// state fits a second time, as an operand, are on the faster kernels of generic_split.cu: here it is K = 256, d = 128 and the like.  Those of generic.cu keep
// every number in fp32, and so do these: the state, the weights and the gradients' partial sums are fp32 in registers and
// shared memory, and a product with such an operand is two mma.sync m16n8k8 tf32 products, of its leading 11 bits and
// of the rest (hi = x rounded to tf32, lo = x - hi: 11 bits, a sign and 11 more); fp16 inputs are exact in tf32.  A product of two
// inputs is one, and goes to m16n8k16 f16 with its operands straight from ldmatrix.  An accumulator inside an mma is
// truncated, which over a chain of them is a bias: 16 terms of a sum are taken from zero, the sums of 16 added in fp32.
// (Share of fp16 results that are not the rounded fp64 value at K = 256, d = 128, 130 tokens, a token at a time / one chain a
// sum / sums of 16: out 0.04 / 0.46 / 0.05 %, gq 0.26 / 0.30 / 0.12, gk 0.13 / 0.33 / 0.10, gv 0.06 / 0.60 / 0.08.  The sums of 16
// cost 1 to 3 % of the time; a third part of 2 bits changes none of these figures and costs 15 %.)  tf32 also has fp32's exponent range, for
// which an fp16 split wants a factor per block and so a place in shared memory.  tcgen05's kind::tf32 would need operands
// padded to its tiles and swizzled and the splits written back to shared memory; at these widths (32 to 256) the warps'
// fragments read straight from fp32 tiles cost less.
//
// A token at a time costs 3.8 us of barriers and shared-memory walks in each of the three kernels (64 heads x 1024 tokens,
// K = 64, d = 32: 11.8 ms forward + backward).  A chunk of C tokens needs the state once (math in rfa.py:57-64, 79-101; S, z
// = sums over all EARLIER tokens, dS, dz over all LATER ones, inv = 1 / max(raw, 1)):
//   forward   P = tril(Q K^T);  raw = rowsum(P) + Q z;  out = inv (P V + Q S);  S += K^T V, z += colsum(K)
//   sweep 1   P, raw as above;  G = g V^T;  W = g S^T;  g.num = rowsum(P o G) + rowsum(Q o W);  gz = -(g.num) inv^2 [raw > 1]
//             gq = inv W + tril(inv G + gz) K + gz z;  S, z as above
//   sweep 2   P' = inv tril(Q K^T);  D = tril(inv G + gz);  gv = P'^T g + K dS;  gk = D^T Q + V dS^T + dz
//             dS += Q^T (inv g), dz += Q^T gz
// Few long sequences are cut into segments (the states at their boundaries: state kernel, then a scan).
//
// A masked product multiplies zeros with the tokens it masks, and 0 * inf is NaN: a chunk whose second operand holds a
// non-finite value takes the masked products element by element, over the unmasked tokens only, so that what a
// token makes of its predecessors never depends on its successors.
#include "generic_mma.cuh"
#include "segments.cuh"
#include "sm100.cuh"

namespace rfa {

constexpr int kGmRegs = 80;      // three CTAs of 256 threads on an SM, or one of 512

// Shared-memory layout (bytes), the same on host and device.  Row pitches: fp16 tiles + 8 and fp32 arrays + 4 elements, which
// keep the fragment reads below (rows 8 apart in g, pairs of columns in t, and their transposes) free of bank conflicts or
// at two ways.
struct GmLayout {
  int Kp, px, py, ps, pp;      // feature rows rounded up to 16 (what the rows from K on hold is never used); pitches of X tiles (q, k), Y tiles (v, g), S and the C x C arrays
  uint32_t x_bytes, y_bytes;   // one tile
  uint32_t S, z, P, D, row, tile, total;
};
// nx / ny: X and Y tiles per stage; cc: C x C arrays; rowf: fp32 per-row arrays
__host__ __device__ inline GmLayout gm_layout(int C, int K, int d, int stages, int nx, int ny, int cc, int rowf) {
  GmLayout L;
  L.Kp = gm_round16(K);
  L.px = L.Kp + 8; L.py = d + 8; L.ps = d + 4; L.pp = C + 4;
  L.x_bytes = (uint32_t)C * L.px * 2; L.y_bytes = (uint32_t)C * L.py * 2;
  L.S = 0;
  L.z = L.S + (uint32_t)L.Kp * L.ps * 4;
  L.P = L.z + (uint32_t)L.Kp * 4;
  L.D = L.P + (cc > 0 ? (uint32_t)C * L.pp * 4 : 0);
  L.row = L.D + (cc > 1 ? (uint32_t)C * L.pp * 4 : 0);
  L.tile = L.row + (uint32_t)rowf * C * 4;
  L.total = L.tile + (uint32_t)stages * (nx * L.x_bytes + ny * L.y_bytes);
  return L;
}
// per-row fp32 arrays of each kernel
__host__ __device__ inline int gm_rows_fwd(int C) { return C / 16 + 1; }                                   // rs, qz
__host__ __device__ inline int gm_rows_bwd_q(int C, int K) { return 2 * (C / 16) + gm_groups32(K) + 3; }   // rs, pg, wq, qz, inv, gz
constexpr int kGmRowsKv = 2, kGmRowsState = 2;                                                             // inv, gz

__device__ __forceinline__ void gm_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Rounding by integer: the conversion unit takes a quarter of the ALU's rate.  The mma drops the low 13 bits of lo.
__device__ __forceinline__ void gm_split(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u;
  lo = __float_as_uint(x - __uint_as_float(hi)) + 0x1000u;
  if (!(fabsf(x) < CUDART_INF_F)) { hi = __float_as_uint(x); lo = 0u; }      // infinities and NaN stay what they are
}
// acc (16 x 8 NT) += sum over l in [l0, l1) of A(i, l) B(l, j) (the outer loop: see the head of the file), one operand exact in tf32 and the other (SPLIT_A: A, else B) in two
// parts.  The sum's order is free, so that slots t and t + 4 of a fragment's inner index stand for l = 2t and 2t + 1: a pair is one
// 8-byte read of an fp32 operand stored along l, and one 8 x 8 block of ldmatrix (two halves a lane) of an fp16 operand,
// whichever way it is stored (trans).  fa(l, a): A at rows g, g + 8 of column l + 2t, then of l + 2t + 1.  fb(l, b): b[n] = B at rows
// l + 2t, l + 2t + 1 of column g of the n-th block of 8.
template <int NT, bool SPLIT_A, int TERMS = 16, class FA, class FB>
__device__ __forceinline__ void gm_product(float (&acc)[NT][4], int nt, int l0, int l1, FA fa, FB fb) {
  const auto step = [&](int l, float (&part)[NT][4]) {
    float x[4];
    float2 b[NT];
    fa(l, x);
    fb(l, b);
    uint32_t a[4], al[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (SPLIT_A) gm_split(x[e], a[e], al[e]);
      else a[e] = __float_as_uint(x[e]);
#pragma unroll
    for (int n = 0; n < NT; ++n)
      if (n < nt) {
        if (SPLIT_A) {
          gm_mma(part[n], al, __float_as_uint(b[n].x), __float_as_uint(b[n].y));
          gm_mma(part[n], a, __float_as_uint(b[n].x), __float_as_uint(b[n].y));
        } else {
          uint32_t h0, l0_, h1, l1_;
          gm_split(b[n].x, h0, l0_); gm_split(b[n].y, h1, l1_);
          gm_mma(part[n], a, l0_, l1_);
          gm_mma(part[n], a, h0, h1);
        }
      }
  };
  for (int l = l0; l < l1; l += TERMS) {
    float part[NT][4] = {};
    step(l, part);
    if (TERMS == 16 && l + 8 < l1) step(l + 8, part);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[n][e] += part[n][e];
  }
}
// operand readers for it
__device__ __forceinline__ void gm_ldsm2(uint32_t (&r)[2], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void gm_ldsm2_t(uint32_t (&r)[2], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ float2 gm_f2(uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); }
__device__ __forceinline__ void gm_pairs(float (&a)[4], float2 x, float2 y) { a[0] = x.x; a[1] = y.x; a[2] = x.y; a[3] = y.y; }
// A = 16 rows of an fp16 tile from row i0
__device__ __forceinline__ auto gm_a_rows(GmTile x, int i0) {
  const int lane = threadIdx.x & 31;
  const __half* p = x.p + (i0 + (lane & 15)) * x.pitch;
  return [=](int l, float (&a)[4]) { uint32_t r[2]; gm_ldsm2(r, p + l); gm_pairs(a, gm_f2(r[0]), gm_f2(r[1])); };
}
// A = 16 columns of an fp16 tile from column i0, transposed
__device__ __forceinline__ auto gm_a_cols(GmTile x, int i0) {
  const int lane = threadIdx.x & 31, pitch = x.pitch;
  const __half* p = x.p + (lane & 7) * pitch + i0 + ((lane >> 3) & 1) * 8;
  return [=](int l, float (&a)[4]) { uint32_t r[2]; gm_ldsm2_t(r, p + l * pitch); gm_pairs(a, gm_f2(r[0]), gm_f2(r[1])); };
}
// A = 16 rows / columns (transposed) of an fp32 array
__device__ __forceinline__ auto gm_a_frows(const float* s, int pitch, int i0) {
  const int lane = threadIdx.x & 31;
  const float *p = s + (i0 + (lane >> 2)) * pitch + 2 * (lane & 3), *q = p + 8 * pitch;
  return [=](int l, float (&a)[4]) { gm_pairs(a, *reinterpret_cast<const float2*>(p + l), *reinterpret_cast<const float2*>(q + l)); };
}
__device__ __forceinline__ auto gm_a_fcols(const float* s, int pitch, int i0) {
  const int lane = threadIdx.x & 31;
  const float* p = s + 2 * (lane & 3) * pitch + i0 + (lane >> 2);
  return [=](int l, float (&a)[4]) { const float* u = p + l * pitch; a[0] = u[0]; a[1] = u[8]; a[2] = u[pitch]; a[3] = u[pitch + 8]; };
}
// B = nt blocks of 8 columns of an fp16 tile from column j0 (blocks from nt on are not read)
template <int NT>
__device__ __forceinline__ auto gm_b_cols(GmTile y, int j0, int nt) {
  const int lane = threadIdx.x & 31, pitch = y.pitch, blk = (lane >> 3) & (NT - 1);
  const __half* p = y.p + (lane & 7) * pitch + j0 + (blk < nt ? blk * 8 : 0);
  return [=](int l, float2 (&b)[NT]) {
    if constexpr (NT == 4) {
      uint32_t r[4];
      gm_ldsm_t(r, p + l * pitch);
#pragma unroll
      for (int n = 0; n < 4; ++n) b[n] = gm_f2(r[n]);
    } else {
      uint32_t r[2];
      gm_ldsm2_t(r, p + l * pitch);
      b[0] = gm_f2(r[0]); b[1] = gm_f2(r[1]);
    }
  };
}
// B = columns from j0 of an fp32 array / of its transpose
template <int NT>
__device__ __forceinline__ auto gm_b_fcols(const float* s, int pitch, int j0, int nt) {
  const int lane = threadIdx.x & 31;
  const float* p = s + 2 * (lane & 3) * pitch + j0 + (lane >> 2);
  return [=](int l, float2 (&b)[NT]) {
    const float* u = p + l * pitch;
#pragma unroll
    for (int n = 0; n < NT; ++n) b[n] = n < nt ? make_float2(u[8 * n], u[pitch + 8 * n]) : make_float2(0.f, 0.f);
  };
}
template <int NT>
__device__ __forceinline__ auto gm_b_frows(const float* s, int pitch, int j0, int nt) {
  const int lane = threadIdx.x & 31;
  const float* p = s + (j0 + (lane >> 2)) * pitch + 2 * (lane & 3);
  return [=](int l, float2 (&b)[NT]) {
#pragma unroll
    for (int n = 0; n < NT; ++n) b[n] = n < nt ? *reinterpret_cast<const float2*>(p + 8 * n * pitch + l) : make_float2(0.f, 0.f);
  };
}
// ---- shared steps ------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void gm_state_in(float* S, float* z, const GmLayout& L, const float* s_in, const float* z_in, int K, int d) {
  for (int e = threadIdx.x; e < L.Kp * d; e += blockDim.x) {
    const int kk = e / d, n = e - kk * d;
    S[kk * L.ps + n] = s_in && kk < K ? s_in[(size_t)kk * d + n] : 0.f;
  }
  for (int i = threadIdx.x; i < L.Kp; i += blockDim.x) z[i] = z_in && i < K ? z_in[i] : 0.f;
}
__device__ __forceinline__ void gm_state_out(const float* S, const float* z, const GmLayout& L, float* s_out, float* z_out, int K, int d) {
  for (int e = threadIdx.x; e < K * d; e += blockDim.x) {
    const int kk = e / d, n = e - kk * d;
    s_out[e] = S[kk * L.ps + n];
  }
  for (int i = threadIdx.x; i < K; i += blockDim.x) z_out[i] = z[i];
}
// S += X^T (wy Y), z += X^T wz over a chunk: summed in registers from zero, then added to the fp32 state with one rounding.
// WEIGHTED: per-row factors inv (of Y) and gz (of z); else 1.
template <int C, bool WEIGHTED>
__device__ __forceinline__ void gm_update(float* S, float* z, const GmLayout& L, GmTile x, GmTile y, const float* inv, const float* gz, int d) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int ng = (d + 8 + 15) / 16, mt = L.Kp / 16;                 // columns d..d+7 stand for z (only d is used)
  for (int w = warp; w < mt * ng; w += blockDim.x >> 5) {
    const int i0 = (w / ng) * 16, j0 = (w % ng) * 16, nt = min(2, (d + 8 - j0) / 8);
    float acc[2][4];
    gm_zero(acc);
    if constexpr (WEIGHTED) {
      const auto cols = gm_b_cols<2>(y, min(j0, d - 8), min(2, (d - j0) / 8));       // the z block is overwritten below
      const auto weighted = [&](int l, float2(&b)[2]) {
        cols(l, b);
        const float2 wi = gm_frow(inv, 0, 0, l + 2 * t), wz = gm_frow(gz, 0, 0, l + 2 * t);
#pragma unroll
        for (int n = 0; n < 2; ++n)
          if (j0 + 8 * n < d) { b[n].x *= wi.x; b[n].y *= wi.y; }
          else b[n] = g == 0 ? wz : make_float2(0.f, 0.f);
      };
      const auto rows = gm_a_cols(x, i0);
      // sums of 8: an fp32 result, whose error at 16 tokens sums of 16 put at 1.0e-7 (a token at a time 8.3e-8, these 6.2e-8)
      gm_product<2, false, 8>(acc, nt, 0, C, rows, weighted);
    } else {
      const __half *pa = x.p + i0 + gm_off_b(lane, x.pitch), *pb = y.p + j0 + gm_off_a(lane, y.pitch);
      const uint32_t ones = g == 0 ? 0x3C003C00u : 0u;         // column d of the z block
#pragma unroll
      for (int l = 0; l < C; l += 16) {
        uint32_t a[4], b[4];
        gm_ldsm_t(a, pa + l * x.pitch);
        if (j0 < d) gm_ldsm_t(b, pb + l * y.pitch);
        else b[0] = b[1] = ones;
        if (j0 + 8 >= d) b[2] = b[3] = ones;
        float part[2][4];
        gm_zero(part);
        gm_mma16(part[0], a, b[0], b[1]);
        if (nt > 1) gm_mma16(part[1], a, b[2], b[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) { acc[0][e] += part[0][e]; acc[1][e] += part[1][e]; }
      }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int j = j0 + 8 * n + 2 * t;
      if (n >= nt) continue;
      if (j < d) {
        float2* p0 = reinterpret_cast<float2*>(S + (i0 + g) * L.ps + j);
        float2* p1 = reinterpret_cast<float2*>(S + (i0 + g + 8) * L.ps + j);
        const float2 u0 = *p0, u1 = *p1;
        *p0 = make_float2(u0.x + acc[n][0], u0.y + acc[n][1]);
        *p1 = make_float2(u1.x + acc[n][2], u1.y + acc[n][3]);
      } else if (j == d) {
        z[i0 + g] += acc[n][0];
        z[i0 + g + 8] += acc[n][2];
      }
    }
  }
}
// ===========================================================================================================================
// forward.  grid (BH, nseg); s_seg / z_seg: the state entering each segment (null = zero)
// ===========================================================================================================================
template <int C, int STAGES>
__global__ void __maxnreg__(kGmRegs)
gm_causal_fwd_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, __half* __restrict__ out,
                     const float* __restrict__ s_seg, const float* __restrict__ z_seg, float* __restrict__ s_out, float* __restrict__ z_out,
                     float* __restrict__ den_out, int64_t T, int BH, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gm_raw[];
  const GmLayout L = gm_layout(C, K, d, STAGES, 2, 1, 1, gm_rows_fwd(C));
  float *S = (float*)(gm_raw + L.S), *z = (float*)(gm_raw + L.z), *P = (float*)(gm_raw + L.P), *rs = (float*)(gm_raw + L.row),
        *qz = rs + (C / 16) * C;
  const int bh = blockIdx.x, seg = blockIdx.y, nseg = gridDim.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = (int)((t_end - t_begin + C - 1) / C);
  const size_t slot = (size_t)bh * nseg + seg;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, pp = L.pp;
  auto tile = [&](int c, int which) {       // 0 q, 1 k, 2 v
    unsigned char* b = gm_raw + L.tile + (uint32_t)(STAGES == 2 ? c & 1 : 0) * (2 * L.x_bytes + L.y_bytes);
    return GmTile{(const __half*)(b + which * L.x_bytes), which < 2 ? L.px : L.py};
  };
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {
    if (c < nchunk) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(c, 0).p, L.px, q, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 1).p, L.px, k, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 2).p, L.py, v, C, d, walk_y, t0, valid, BH, bh, nullptr);
    }
    gm_commit();
  };
  for (int s = 0; s < STAGES; ++s)
    for (int i = 0; i < 3; ++i) gm_pad(tile(s, i), C, i < 2 ? K : d);
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(0);
  gm_state_in(S, z, L, s_seg ? s_seg + slot * K * d : nullptr, z_seg ? z_seg + slot * K : nullptr, K, d);
  for (int c = 0; c < nchunk; ++c) {
    if (c == nchunk - 1) sm100::pdl_launch_dependents();
    if (STAGES == 2) { load(c + 1); gm_wait<1>(); } else gm_wait<0>();
    const GmTile tq = tile(c, 0), tk = tile(c, 1), tv = tile(c, 2);
    const int64_t t0 = t_begin + (int64_t)c * C;
    const int valid = (int)min((int64_t)C, t_end - t0);
    const bool odd = __syncthreads_or(gm_odd(tv.p, tv.pitch, C, walk_y)) != 0;
    // P = tril(Q K^T), its row sums per 16 columns, q . z
    constexpr int MT = C / 16;
    for (int w = warp; w < MT * MT; w += blockDim.x >> 5) {
      const int mi = w / MT, ni = w % MT, i0 = mi * 16, j0 = ni * 16;
      if (ni > mi) continue;
      float acc[2][4];
      gm_zero(acc);
      gm_exact(acc, tq, i0, tk, j0, K);
      float r0 = 0.f, r1 = 0.f;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int j = j0 + 8 * n + 2 * t, i = i0 + g;
        if (j > i) acc[n][0] = 0.f;
        if (j + 1 > i) acc[n][1] = 0.f;
        if (j > i + 8) acc[n][2] = 0.f;
        if (j + 1 > i + 8) acc[n][3] = 0.f;
        *reinterpret_cast<float2*>(P + i * L.pp + j) = make_float2(acc[n][0], acc[n][1]);
        *reinterpret_cast<float2*>(P + (i + 8) * L.pp + j) = make_float2(acc[n][2], acc[n][3]);
        r0 += acc[n][0] + acc[n][1];
        r1 += acc[n][2] + acc[n][3];
      }
      r0 = gm_quad(r0); r1 = gm_quad(r1);
      if (t == 0) { rs[ni * C + i0 + g] = r0; rs[ni * C + i0 + g + 8] = r1; }
    }
    gm_qz<C>(qz, tq, z, K);
    __syncthreads();
    // out = (P V + Q S) / max(raw, 1)
    const int ng = (d + 15) / 16;
    for (int w = warp; w < MT * ng; w += blockDim.x >> 5) {
      const int mi = w / ng, i0 = mi * 16, j0 = (w % ng) * 16, nt = min(2, (d - j0) / 8);
      float acc[2][4];
      gm_zero(acc);
      auto la = [=](int i, int l) { return gm_frow(P, pp, i, l); };
      auto lb = [=](int l, int j) { return gm_col(tv, l, j); };
      if (odd) gm_product_masked<2>(acc, i0, j0, nt, 0, i0 + 16, la, lb, [](int i, int l) { return l <= i; });
      else gm_product<2, true>(acc, nt, 0, i0 + 16, gm_a_frows(P, pp, i0), gm_b_cols<2>(tv, j0, nt));
      gm_product<2, false>(acc, nt, 0, K, gm_a_rows(tq, i0), gm_b_fcols<2>(S, L.ps, j0, nt));
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
    if (c + 1 < nchunk || s_out) gm_update<C, false>(S, z, L, tk, tv, nullptr, nullptr, d);
    __syncthreads();
    if (STAGES == 1) load(c + 1);
  }
  if (s_out && seg == nseg - 1) {
    if (nchunk == 0) __syncthreads();
    gm_state_out(S, z, L, s_out + (size_t)bh * K * d, z_out + (size_t)bh * K, K, d);
  }
}

// ===========================================================================================================================
// backward, sweep 1: gq, raw denominators, gz
// ===========================================================================================================================
template <int C, int STAGES>
__global__ void __maxnreg__(kGmRegs)
gm_causal_bwd_q_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, const __half* __restrict__ gr,
                       __half* __restrict__ gq, const float* __restrict__ s_seg, const float* __restrict__ z_seg,
                       float* __restrict__ ws_den, float* __restrict__ ws_gz, int64_t T, int BH, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gm_raw[];
  const GmLayout L = gm_layout(C, K, d, STAGES, 2, 2, 1, gm_rows_bwd_q(C, K));
  constexpr int MT = C / 16;
  const int kg = gm_groups32(K);
  float *S = (float*)(gm_raw + L.S), *z = (float*)(gm_raw + L.z), *G = (float*)(gm_raw + L.P), *rs = (float*)(gm_raw + L.row),
        *pg = rs + MT * C, *wq = pg + MT * C, *qz = wq + kg * C, *inv = qz + C, *gz = inv + C;
  const int bh = blockIdx.x, seg = blockIdx.y, nseg = gridDim.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = (int)((t_end - t_begin + C - 1) / C);
  const size_t slot = (size_t)bh * nseg + seg;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, pp = L.pp;
  auto tile = [&](int c, int which) {       // 0 q, 1 k, 2 v, 3 g
    unsigned char* b = gm_raw + L.tile + (uint32_t)(STAGES == 2 ? c & 1 : 0) * (2 * L.x_bytes + 2 * L.y_bytes);
    return GmTile{(const __half*)(b + (which < 2 ? which * L.x_bytes : 2 * L.x_bytes + (which - 2) * L.y_bytes)), which < 2 ? L.px : L.py};
  };
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {
    if (c < nchunk) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(c, 0).p, L.px, q, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 1).p, L.px, k, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 2).p, L.py, v, C, d, walk_y, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 3).p, L.py, gr, C, d, walk_y, t0, valid, BH, bh, nullptr);
    }
    gm_commit();
  };
  for (int s = 0; s < STAGES; ++s)
    for (int i = 0; i < 4; ++i) gm_pad(tile(s, i), C, i < 2 ? K : d);
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(0);
  gm_state_in(S, z, L, s_seg ? s_seg + slot * K * d : nullptr, z_seg ? z_seg + slot * K : nullptr, K, d);
  for (int c = 0; c < nchunk; ++c) {
    if (c == nchunk - 1) sm100::pdl_launch_dependents();
    if (STAGES == 2) { load(c + 1); gm_wait<1>(); } else gm_wait<0>();
    const GmTile tq = tile(c, 0), tk = tile(c, 1), tv = tile(c, 2), tg = tile(c, 3);
    const int64_t t0 = t_begin + (int64_t)c * C;
    const int valid = (int)min((int64_t)C, t_end - t0);
    const bool odd = __syncthreads_or(gm_odd(tk.p, tk.pitch, C, walk_x)) != 0;
    // G = g V^T on and below the diagonal; per 16 columns the row sums of P and of P o G
    for (int w = warp; w < MT * MT; w += blockDim.x >> 5) {
      const int mi = w / MT, ni = w % MT, i0 = mi * 16, j0 = ni * 16;
      if (ni > mi) continue;
      float p[2][4], a[2][4];
      gm_zero(p); gm_zero(a);
      gm_exact(p, tq, i0, tk, j0, K);
      gm_exact(a, tg, i0, tv, j0, d);
      float r[2] = {0.f, 0.f}, s[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = j0 + 8 * n + 2 * t + (e & 1), i = i0 + g + 8 * (e >> 1);
          if (j <= i) { r[e >> 1] += p[n][e]; s[e >> 1] = fmaf(p[n][e], a[n][e], s[e >> 1]); }
        }
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int j = j0 + 8 * n + 2 * t;
        *reinterpret_cast<float2*>(G + (i0 + g) * L.pp + j) = make_float2(a[n][0], a[n][1]);
        *reinterpret_cast<float2*>(G + (i0 + g + 8) * L.pp + j) = make_float2(a[n][2], a[n][3]);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        r[e] = gm_quad(r[e]); s[e] = gm_quad(s[e]);
        if (t == 0) { rs[ni * C + i0 + g + 8 * e] = r[e]; pg[ni * C + i0 + g + 8 * e] = s[e]; }
      }
    }
    // W = g S^T: the row sums of Q o W per 32 features
    for (int w = warp; w < MT * kg; w += blockDim.x >> 5) {
      const int i0 = (w / kg) * 16, gi = w % kg, j0 = gi * 32, nt = min(4, (K - j0) / 8);
      float a[4][4];
      gm_zero(a);
      gm_product<4, false>(a, nt, 0, d, gm_a_rows(tg, i0), gm_b_frows<4>(S, L.ps, j0, nt));
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
    if (threadIdx.x < C) {
      const int i = threadIdx.x;
      float raw = qz[i], gn = 0.f;
      for (int b = 0; b <= i / 16; ++b) { raw += rs[b * C + i]; gn += pg[b * C + i]; }
      for (int b = 0; b < kg; ++b) gn += wq[b * C + i];
      const float iv = 1.f / fmaxf(raw, kEps);
      inv[i] = iv;
      gz[i] = raw > kEps ? -gn * iv * iv : 0.f;                    // strict >, upstream rfa.py:91
      if (i < valid) { ws_den[(size_t)bh * T + t0 + i] = raw; ws_gz[(size_t)bh * T + t0 + i] = gz[i]; }
    }
    __syncthreads();
    // gq = inv W + tril(inv G + gz) K + gz z
    for (int w = warp; w < MT * kg; w += blockDim.x >> 5) {
      const int i0 = (w / kg) * 16, j0 = (w % kg) * 32, nt = min(4, (K - j0) / 8);
      float a[4][4];
      gm_zero(a);
      gm_product<4, false>(a, nt, 0, d, gm_a_rows(tg, i0), gm_b_frows<4>(S, L.ps, j0, nt));
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[n][e] *= inv[i0 + g + 8 * (e >> 1)];
      auto la = [=](int i, int l) {
        const float2 u = gm_frow(G, pp, i, l);
        return make_float2(l <= i ? fmaf(inv[i], u.x, gz[i]) : 0.f, l + 1 <= i ? fmaf(inv[i], u.y, gz[i]) : 0.f);
      };
      auto lb = [=](int l, int j) { return gm_col(tk, l, j); };
      if (odd) gm_product_masked<4>(a, i0, j0, nt, 0, i0 + 16, la, lb, [](int i, int l) { return l <= i; });
      else gm_product<4, true>(a, nt, 0, i0 + 16, [&](int l, float(&u)[4]) { gm_pairs(u, la(i0 + g, l + 2 * t), la(i0 + g + 8, l + 2 * t)); },
                               gm_b_cols<4>(tk, j0, nt));
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
    if (c + 1 < nchunk) gm_update<C, false>(S, z, L, tk, tv, nullptr, nullptr, d);
    __syncthreads();
    if (STAGES == 1) load(c + 1);
  }
}

// ===========================================================================================================================
// backward, sweep 2 (chunks in reverse): gk, gv
// ===========================================================================================================================
template <int C, int STAGES>
__global__ void __maxnreg__(kGmRegs)
gm_causal_bwd_kv_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, const __half* __restrict__ gr,
                        __half* __restrict__ gk, __half* __restrict__ gv, const float* __restrict__ ws_den, const float* __restrict__ ws_gz,
                        const float* __restrict__ ds_seg, const float* __restrict__ dz_seg, int64_t T, int BH, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gm_raw[];
  const GmLayout L = gm_layout(C, K, d, STAGES, 2, 2, 2, kGmRowsKv);
  constexpr int MT = C / 16;
  const int kg = gm_groups32(K);
  float *S = (float*)(gm_raw + L.S), *z = (float*)(gm_raw + L.z), *P = (float*)(gm_raw + L.P), *D = (float*)(gm_raw + L.D),
        *inv = (float*)(gm_raw + L.row), *gz = inv + C;
  const int bh = blockIdx.x, seg = blockIdx.y, nseg = gridDim.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = (int)((t_end - t_begin + C - 1) / C);
  const size_t slot = (size_t)bh * nseg + seg;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, pp = L.pp;
  auto tile = [&](int c, int which) {       // 0 q, 1 k, 2 v, 3 g
    unsigned char* b = gm_raw + L.tile + (uint32_t)(STAGES == 2 ? c & 1 : 0) * (2 * L.x_bytes + 2 * L.y_bytes);
    return GmTile{(const __half*)(b + (which < 2 ? which * L.x_bytes : 2 * L.x_bytes + (which - 2) * L.y_bytes)), which < 2 ? L.px : L.py};
  };
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {                   // c counts down to 0
    if (c >= 0) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(c, 0).p, L.px, q, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 1).p, L.px, k, C, K, walk_x, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 2).p, L.py, v, C, d, walk_y, t0, valid, BH, bh, nullptr);
      gm_load((__half*)tile(c, 3).p, L.py, gr, C, d, walk_y, t0, valid, BH, bh, nullptr);
    }
    gm_commit();
  };
  for (int s = 0; s < STAGES; ++s)
    for (int i = 0; i < 4; ++i) gm_pad(tile(s, i), C, i < 2 ? K : d);
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(nchunk - 1);
  gm_state_in(S, z, L, ds_seg ? ds_seg + slot * K * d : nullptr, dz_seg ? dz_seg + slot * K : nullptr, K, d);
  for (int c = nchunk - 1; c >= 0; --c) {
    if (c == 0) sm100::pdl_launch_dependents();
    const int64_t t0 = t_begin + (int64_t)c * C;
    const int valid = (int)min((int64_t)C, t_end - t0);
    gm_row_scalars(inv, gz, ws_den, ws_gz, C, (size_t)bh * T + t0, valid);
    if (STAGES == 2) { load(c - 1); gm_wait<1>(); } else gm_wait<0>();
    const GmTile tq = tile(c, 0), tk = tile(c, 1), tv = tile(c, 2), tg = tile(c, 3);
    const bool odd = __syncthreads_or(gm_odd(tq.p, tq.pitch, C, walk_x) || gm_odd(tg.p, tg.pitch, C, walk_y)) != 0;
    // P' = inv tril(Q K^T), D = tril(inv g V^T + gz)
    for (int w = warp; w < MT * MT; w += blockDim.x >> 5) {
      const int mi = w / MT, ni = w % MT, i0 = mi * 16, j0 = ni * 16;
      if (ni > mi) continue;
      float p[2][4], a[2][4];
      gm_zero(p); gm_zero(a);
      gm_exact(p, tq, i0, tk, j0, K);
      gm_exact(a, tg, i0, tv, j0, d);
#pragma unroll
      for (int n = 0; n < 2; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int j = j0 + 8 * n + 2 * t + (e & 1), i = i0 + g + 8 * (e >> 1);
          p[n][e] = j <= i ? p[n][e] * inv[i] : 0.f;
          a[n][e] = j <= i ? fmaf(a[n][e], inv[i], gz[i]) : 0.f;
        }
        const int j = j0 + 8 * n + 2 * t, i = i0 + g;
        *reinterpret_cast<float2*>(P + i * L.pp + j) = make_float2(p[n][0], p[n][1]);
        *reinterpret_cast<float2*>(P + (i + 8) * L.pp + j) = make_float2(p[n][2], p[n][3]);
        *reinterpret_cast<float2*>(D + i * L.pp + j) = make_float2(a[n][0], a[n][1]);
        *reinterpret_cast<float2*>(D + (i + 8) * L.pp + j) = make_float2(a[n][2], a[n][3]);
      }
    }
    __syncthreads();
    // gk = D^T Q + V dS^T + dz   and   gv = P'^T g + K dS
    const int ng = (d + 15) / 16;
    for (int w = warp; w < MT * (kg + ng); w += blockDim.x >> 5) {
      if (w < MT * kg) {
        const int i0 = (w / kg) * 16, j0 = (w % kg) * 32, nt = min(4, (K - j0) / 8);
        float a[4][4];
        gm_zero(a);
        auto la = [=](int i, int l) { return gm_fcol(D, pp, l, i); };
        auto lb = [=](int l, int j) { return gm_col(tq, l, j); };
        if (odd) gm_product_masked<4>(a, i0, j0, nt, i0, C, la, lb, [](int i, int l) { return l >= i; });
        else gm_product<4, true>(a, nt, i0, C, gm_a_fcols(D, pp, i0), gm_b_cols<4>(tq, j0, nt));
        gm_product<4, false>(a, nt, 0, d, gm_a_rows(tv, i0), gm_b_frows<4>(S, L.ps, j0, nt));
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
        const int u = w - MT * kg, i0 = (u / ng) * 16, j0 = (u % ng) * 16, nt = min(2, (d - j0) / 8);
        float a[2][4];
        gm_zero(a);
        auto la = [=](int i, int l) { return gm_fcol(P, pp, l, i); };
        auto lb = [=](int l, int j) { return gm_col(tg, l, j); };
        if (odd) gm_product_masked<2>(a, i0, j0, nt, i0, C, la, lb, [](int i, int l) { return l >= i; });
        else gm_product<2, true>(a, nt, i0, C, gm_a_fcols(P, pp, i0), gm_b_cols<2>(tg, j0, nt));
        gm_product<2, false>(a, nt, 0, K, gm_a_rows(tk, i0), gm_b_fcols<2>(S, L.ps, j0, nt));
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
    if (c > 0) gm_update<C, true>(S, z, L, tq, tg, inv, gz, d);
    __syncthreads();
    if (STAGES == 1) load(c - 1);
  }
}

// ===========================================================================================================================
// state reduction over runs of tokens: sum x (x) y, sum x (padded keys left out), or with ws_den / ws_gz the reverse one,
// sum x (x) (inv y), sum gz x.  grid (BH, runs <= nseg)
// ===========================================================================================================================
template <int C, int STAGES, bool WEIGHTED>
__global__ void __maxnreg__(kGmRegs)
gm_state_kernel(const __half* __restrict__ x, const __half* __restrict__ y, const uint8_t* __restrict__ pad_mask,
                const float* __restrict__ ws_den, const float* __restrict__ ws_gz, float* __restrict__ s_out, float* __restrict__ z_out,
                int64_t T, int BH, int H, int nseg, int64_t tseg, int K, int d) {
  extern __shared__ __align__(16) unsigned char gm_raw[];
  const GmLayout L = gm_layout(C, K, d, STAGES, 1, 1, 0, kGmRowsState);
  float *S = (float*)(gm_raw + L.S), *z = (float*)(gm_raw + L.z), *inv = (float*)(gm_raw + L.row), *gz = inv + C;
  const int bh = blockIdx.x, seg = blockIdx.y;
  const int64_t t_begin = seg * tseg, t_end = min(T, t_begin + tseg);
  const int nchunk = t_end > t_begin ? (int)((t_end - t_begin + C - 1) / C) : 0;
  const size_t slot = (size_t)bh * nseg + seg;
  const uint8_t* mrow = pad_mask ? pad_mask + (size_t)(bh / H) * T : nullptr;
  auto tile = [&](int c, int which) {
    unsigned char* b = gm_raw + L.tile + (uint32_t)(STAGES == 2 ? c & 1 : 0) * (L.x_bytes + L.y_bytes);
    return GmTile{(const __half*)(b + which * L.x_bytes), which < 1 ? L.px : L.py};
  };
  const GmWalk walk_x = gm_walk(K), walk_y = gm_walk(d);
  auto load = [&](int c) {
    if (c < nchunk) {
      const int64_t t0 = t_begin + (int64_t)c * C;
      const int valid = (int)min((int64_t)C, t_end - t0);
      gm_load((__half*)tile(c, 0).p, L.px, x, C, K, walk_x, t0, valid, BH, bh, mrow);
      gm_load((__half*)tile(c, 1).p, L.py, y, C, d, walk_y, t0, valid, BH, bh, mrow);
    }
    gm_commit();
  };
  sm100::pdl_wait();            // everything above overlaps the tail of the previous kernel in the stream
  load(0);
  gm_state_in(S, z, L, nullptr, nullptr, K, d);
  for (int c = 0; c < nchunk; ++c) {
    if (c == nchunk - 1) sm100::pdl_launch_dependents();
    const int64_t t0 = t_begin + (int64_t)c * C;
    if (WEIGHTED) gm_row_scalars(inv, gz, ws_den, ws_gz, C, (size_t)bh * T + t0, (int)min((int64_t)C, t_end - t0));
    if (STAGES == 2) { load(c + 1); gm_wait<1>(); } else gm_wait<0>();
    __syncthreads();
    gm_update<C, WEIGHTED>(S, z, L, tile(c, 0), tile(c, 1), inv, gz, d);
    __syncthreads();
    if (STAGES == 1) load(c + 1);
  }
  if (nchunk == 0) __syncthreads();
  gm_state_out(S, z, L, s_out + slot * K * d, z_out + slot * K, K, d);
}

// ---------------------------------------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------------------------------------
constexpr uint32_t kGmSmemMax = 227 * 1024;

// the most shared memory one of the three causal kernels takes
static uint32_t gm_need(int C, int stages, int K, int d) {
  const uint32_t a = gm_layout(C, K, d, stages, 2, 2, 1, gm_rows_bwd_q(C, K)).total, b = gm_layout(C, K, d, stages, 2, 2, 2, kGmRowsKv).total;
  return a > b ? a : b;
}
struct GmShape { int C, stages, ctas, threads; };
// The longest chunk that fits, two stages before one: a longer chunk shares the state's products and the barriers among
// more tokens.  C = 0: nothing fits.  A chunk's phases are chains of latencies, so that an SM wants 16 warps or more: from several
// CTAs of 256 threads (up to 3), or from one of 512 where the state leaves room for one (K = 256, d = 128, 64 heads x 512
// tokens, backward: 740 us with 256).
static GmShape gm_shape(int K, int d) {
  for (int C : {64, 32, 16})
    for (int stages : {2, 1})
      if (const uint32_t need = gm_need(C, stages, K, d); need <= kGmSmemMax) {
        const int n = (int)(kGmSmemMax / (need + 1024));
        return GmShape{C, stages, n < 1 ? 1 : n > 3 ? 3 : n, n < 2 ? 512 : 256};
      }
  return GmShape{0, 0, 0, 0};
}

// the kernels whose operands are split into fp16 tiles once (generic_split.cu), where they fit
int split_chunk(int64_t T, int BH, int K, int d, bool whole, int* ctas);
int launch_causal_split_fwd(const __half* q, const __half* k, const __half* v, __half* out, const float* s_seg, const float* z_seg, float* s_out,
                            float* z_out, float* den_out, int64_t T, int BH, int nseg, int64_t tseg, int K, int d, cudaStream_t st);
int launch_causal_split_bwd_q(const __half* q, const __half* k, const __half* v, const __half* g, __half* gq, const float* s_seg, const float* z_seg,
                              float* ws_den, float* ws_gz, int64_t T, int BH, int nseg, int64_t tseg, int K, int d, cudaStream_t st);
int launch_causal_split_bwd_kv(const __half* q, const __half* k, const __half* v, const __half* g, __half* gk, __half* gv, const float* ws_den,
                               const float* ws_gz, const float* ds_seg, const float* dz_seg, int64_t T, int BH, int nseg, int64_t tseg, int K,
                               int d, cudaStream_t st);
int launch_state_split(const __half* x, const __half* y, const uint8_t* pad_mask, const float* ws_den, const float* ws_gz, float* s, float* z,
                       int64_t T, int BH, int H, int nseg, int64_t tseg, int runs, int K, int d, cudaStream_t st);

// Whether those take the call.  Where only their chunks of 16 fit, one CTA makes a 16 x 16 block of scores at a time, and the longer chunks here
// are faster as soon as several follow one another: a token here costs 7/8 of one there (half of it at d = 8, which is padded to 16
// there), a call one chunk of 16 more.  us forward + backward, here / there: (160, 128), 8 heads x 512 tokens 152 / 92, 64 x 512 495 / 550,
// 128 x 1024 1519 / 1765; (512, 32) 122 / 99, 644 / 639, 2046 / 2125; (520, 24), 16 x 512 185 / 175; (896, 8), 8 x 64 99 / 60, 8 x 512 110 / 119,
// 64 x 512 722 / 853.
static bool takes_split(int64_t T, int BH, int K, int d, bool whole) {
  int ctas = 1;
  const int chunk = split_chunk(T, BH, K, d, whole, &ctas);
  if (chunk != 16) return chunk > 0;
  const GmShape here = gm_shape(K, d);
  if (here.C <= 16) return true;
  const auto chunks = [&](int C, int n) { return cut_segments(T, C, whole ? 1 : kSms * n / BH, 1).tseg / C; };      // one after another
  return (d < 16 ? 32 : 16) * chunks(16, ctas) < 7 * here.C * chunks(here.C, here.ctas) / 8 + 16;
}

// Tokens per chunk of the chunked kernels for these calls, 0 when the geometry does not fit them; *ctas = how many of their CTAs
// one SM holds.
int generic_chunk(int64_t T, int BH, int K, int d, int* ctas) {
  if (K <= 0 || d <= 0 || K % 8 || d % 8 || K > 1024 || d > 1024) return 0;
  if (takes_split(T, BH, K, d, false)) return split_chunk(T, BH, K, d, false, ctas);
  const GmShape s = gm_shape(K, d);
  if (ctas) *ctas = s.ctas;
  return s.C;
}

template <class KERNEL, class... Args>
static int gm_launch(KERNEL kernel, const char* what, int threads, uint32_t smem, dim3 grid, cudaStream_t st, Args... args) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail((int)e, "%s: cannot reserve %u bytes of shared memory: %s", what, smem, cudaGetErrorString(e));
  sm100::launch_pdl(kernel, grid, dim3(threads), smem, st, args...);      // (K, d) = (256, 128), 32 x 512: 422.6 -> 415.4 us a step, 128 x 512 1115 -> 1107
  return check_launch(what);
}
#define RFA_GM_DISPATCH(shape, CALL)                                  \
  do {                                                                \
    const GmShape gs_ = (shape);                                      \
    if (gs_.C == 64) { CALL(64, 1); }                                 \
    if (gs_.C == 32) { if (gs_.stages == 2) { CALL(32, 2); } else { CALL(32, 1); } } \
    if (gs_.stages == 2) { CALL(16, 2); } else { CALL(16, 1); }       \
  } while (0)

int launch_causal_chunked_fwd(const __half* q, const __half* k, const __half* v, __half* out, const float* s_seg, const float* z_seg,
                              float* s_out, float* z_out, float* den_out, int64_t T, int BH, int nseg, int64_t tseg, int K, int d,
                              cudaStream_t st) {
  if (takes_split(T, BH, K, d, nseg == 1)) return launch_causal_split_fwd(q, k, v, out, s_seg, z_seg, s_out, z_out, den_out, T, BH, nseg, tseg, K, d, st);
#define RFA_GM_CALL(C, N) return gm_launch(gm_causal_fwd_kernel<C, N>, "rfa_causal_fwd (chunked)", gs_.threads, gm_layout(C, K, d, N, 2, 1, 1, gm_rows_fwd(C)).total, \
                                           dim3(BH, nseg), st, q, k, v, out, s_seg, z_seg, s_out, z_out, den_out, T, BH, tseg, K, d)
  RFA_GM_DISPATCH(gm_shape(K, d), RFA_GM_CALL);
#undef RFA_GM_CALL
}

int launch_causal_chunked_bwd_q(const __half* q, const __half* k, const __half* v, const __half* g, __half* gq, const float* s_seg,
                                const float* z_seg, float* ws_den, float* ws_gz, int64_t T, int BH, int nseg, int64_t tseg, int K, int d,
                                cudaStream_t st) {
  if (takes_split(T, BH, K, d, nseg == 1)) return launch_causal_split_bwd_q(q, k, v, g, gq, s_seg, z_seg, ws_den, ws_gz, T, BH, nseg, tseg, K, d, st);
#define RFA_GM_CALL(C, N) return gm_launch(gm_causal_bwd_q_kernel<C, N>, "rfa_causal_bwd_q (chunked)", gs_.threads, gm_layout(C, K, d, N, 2, 2, 1, gm_rows_bwd_q(C, K)).total, \
                                           dim3(BH, nseg), st, q, k, v, g, gq, s_seg, z_seg, ws_den, ws_gz, T, BH, tseg, K, d)
  RFA_GM_DISPATCH(gm_shape(K, d), RFA_GM_CALL);
#undef RFA_GM_CALL
}

int launch_causal_chunked_bwd_kv(const __half* q, const __half* k, const __half* v, const __half* g, __half* gk, __half* gv,
                                 const float* ws_den, const float* ws_gz, const float* ds_seg, const float* dz_seg, int64_t T, int BH,
                                 int nseg, int64_t tseg, int K, int d, cudaStream_t st) {
  if (takes_split(T, BH, K, d, nseg == 1)) return launch_causal_split_bwd_kv(q, k, v, g, gk, gv, ws_den, ws_gz, ds_seg, dz_seg, T, BH, nseg, tseg, K, d, st);
#define RFA_GM_CALL(C, N) return gm_launch(gm_causal_bwd_kv_kernel<C, N>, "rfa_causal_bwd_kv (chunked)", gs_.threads, gm_layout(C, K, d, N, 2, 2, 2, kGmRowsKv).total, \
                                           dim3(BH, nseg), st, q, k, v, g, gk, gv, ws_den, ws_gz, ds_seg, dz_seg, T, BH, tseg, K, d)
  RFA_GM_DISPATCH(gm_shape(K, d), RFA_GM_CALL);
#undef RFA_GM_CALL
}

// the first `runs` of nseg runs of tokens; ws_den / ws_gz null: sums of k (x) v and k; else of q (x) (g / den) and gz q
int launch_state_chunked(const __half* x, const __half* y, const uint8_t* pad_mask, const float* ws_den, const float* ws_gz, float* s,
                         float* z, int64_t T, int BH, int H, int nseg, int64_t tseg, int runs, int K, int d, cudaStream_t st) {
  if (takes_split(T, BH, K, d, nseg == 1)) return launch_state_split(x, y, pad_mask, ws_den, ws_gz, s, z, T, BH, H, nseg, tseg, runs, K, d, st);
#define RFA_GM_CALL(C, N)                                                                                                             \
  return ws_den ? gm_launch(gm_state_kernel<C, N, true>, "state reduction (chunked)", gs_.threads, gm_layout(C, K, d, N, 1, 1, 0, kGmRowsState).total, \
                            dim3(BH, runs), st, x, y, pad_mask, ws_den, ws_gz, s, z, T, BH, H, nseg, tseg, K, d)                             \
                : gm_launch(gm_state_kernel<C, N, false>, "state reduction (chunked)", gs_.threads, gm_layout(C, K, d, N, 1, 1, 0, kGmRowsState).total, \
                            dim3(BH, runs), st, x, y, pad_mask, ws_den, ws_gz, s, z, T, BH, H, nseg, tseg, K, d)
  RFA_GM_DISPATCH(gm_shape(K, d), RFA_GM_CALL);
#undef RFA_GM_CALL
}

}  // namespace rfa
