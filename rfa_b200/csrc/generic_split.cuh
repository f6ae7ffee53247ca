// fp32 matrices as operands of mma.sync m16n8k16 f16: two fp16 tiles and a power of two per 16 x 16 block, or for each of a block's rows or columns
// where they are results that must not lose bits to one another.
//
// x is held as hi = fp16(s x) and lo = fp16(s x - hi): 22 bits.  s takes the block's largest finite element to [2^14, 2^15), so that
// fp16's range costs nothing: an element down to 2^-17 of its block's largest keeps all 22 bits, and what a smaller one loses
// is 2^-39 of the largest, 2^-15 of that one's own rounding in fp32.  A product with an fp16 operand, which is exact, is two mma; of two
// split operands three.  An mma's accumulator truncates, which over a chain is a bias: a sum of 16 terms is taken from zero, small
// parts first, scaled back, and added to the others in fp32.
#pragma once

#include "generic_mma.cuh"

namespace rfa {

// a matrix in two fp16 parts and the factors 1 / s of its 16 x 16 blocks, `sp` of them to a row of blocks
struct GsSplit {
  __half *hi, *lo;
  float* inv_s;
  int pitch, sp;
};

// ---- splitting ---------------------------------------------------------------------------------------------------------------
constexpr uint32_t kGsInf = 0x7F800000u;
__device__ __forceinline__ uint32_t gs_mag(float x) { return __float_as_uint(x) & 0x7FFFFFFFu; }
// s and 1 / s for a block whose largest finite magnitude has these bits; both stay normal numbers
__device__ __forceinline__ void gs_factors(uint32_t mag, float& s, float& inv_s) {
  const uint32_t e = max(mag & kGsInf, 15u << 23);
  s = __uint_as_float((268u << 23) - e);
  inv_s = __uint_as_float(e - (14u << 23));
}
// ODD: infinities and NaN stay what they are, in hi
template <bool ODD>
__device__ __forceinline__ void gs_parts(float x, float y, float s, uint32_t& hi, uint32_t& lo) {
  x *= s; y *= s;
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(!ODD || fabsf(x) < CUDART_INF_F ? x - f.x : 0.f, !ODD || fabsf(y) < CUDART_INF_F ? y - f.y : 0.f);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
template <bool ODD>
__device__ __forceinline__ void gs_put_as(const GsSplit& m, int i0, int j0, const float (&a)[2][4], uint32_t mag) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  float s, inv_s;
  gs_factors(mag, s, inv_s);
  if (lane == 0) m.inv_s[(i0 >> 4) * m.sp + (j0 >> 4)] = inv_s;
  const int at = (i0 + g) * m.pitch + j0 + 2 * t;
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      uint32_t hi, lo;
      gs_parts<ODD>(a[n][2 * r], a[n][2 * r + 1], s, hi, lo);
      *reinterpret_cast<uint32_t*>(m.hi + at + 8 * r * m.pitch + 8 * n) = hi;
      *reinterpret_cast<uint32_t*>(m.lo + at + 8 * r * m.pitch + 8 * n) = lo;
    }
}
static __device__ __noinline__ void gs_put_odd(GsSplit m, int i0, int j0, float4 x, float4 y) {      // by value: arguments stay in registers
  const float a[2][4] = {{x.x, x.y, x.z, x.w}, {y.x, y.y, y.z, y.w}};
  uint32_t mag = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const uint32_t b = gs_mag(a[e >> 2][e & 3]);
    if (b < kGsInf) mag = max(mag, b);
  }
  gs_put_as<true>(m, i0, j0, a, __reduce_max_sync(0xffffffffu, mag));
}
// a block in accumulator layout (a[n]: rows g, g + 8, columns 8 n + 2 t, + 1) -> rows i0.., columns j0.. of m
__device__ __forceinline__ void gs_put(const GsSplit& m, int i0, int j0, const float (&a)[2][4]) {
  uint32_t mag = 0;
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) mag = max(mag, gs_mag(a[n][e]));
  mag = __reduce_max_sync(0xffffffffu, mag);
  if (mag < kGsInf) gs_put_as<false>(m, i0, j0, a, mag);
  else gs_put_odd(m, i0, j0, make_float4(a[0][0], a[0][1], a[0][2], a[0][3]), make_float4(a[1][0], a[1][1], a[1][2], a[1][3]));
}

// ---- with a factor for each row of a block -----------------------------------------------------------------------------------
// For products whose results are of one row each: a row does not lose bits to a larger one beside it.
struct GsByRow {
  __half *hi, *lo;
  float* inv_s;      // [row fr + column / 16 fc]
  int pitch, fr, fc;
};
// the largest (ODD: finite) magnitudes of rows g and g + 8, in all four lanes of a row
template <bool ODD>
__device__ __forceinline__ void gs_row_mags(uint32_t (&mag)[2], const float (&a)[2][4]) {
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    mag[r] = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t b = gs_mag(a[e >> 1][2 * r + (e & 1)]);
      if (!ODD || b < kGsInf) mag[r] = max(mag[r], b);
    }
    mag[r] = max(mag[r], __shfl_xor_sync(0xffffffffu, mag[r], 1));
    mag[r] = max(mag[r], __shfl_xor_sync(0xffffffffu, mag[r], 2));
  }
}
template <bool ODD>
__device__ __forceinline__ void gs_put_rows_as(const GsByRow& m, int i0, int j0, const float (&a)[2][4], const uint32_t (&mag)[2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = i0 + g + 8 * r, at = row * m.pitch + j0 + 2 * t;
    float s, inv_s;
    gs_factors(mag[r], s, inv_s);
    if (t == 0) m.inv_s[row * m.fr + (j0 >> 4) * m.fc] = inv_s;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      uint32_t hi, lo;
      gs_parts<ODD>(a[n][2 * r], a[n][2 * r + 1], s, hi, lo);
      *reinterpret_cast<uint32_t*>(m.hi + at + 8 * n) = hi;
      *reinterpret_cast<uint32_t*>(m.lo + at + 8 * n) = lo;
    }
  }
}
static __device__ __noinline__ void gs_put_rows_odd(GsByRow m, int i0, int j0, float4 x, float4 y) {
  const float a[2][4] = {{x.x, x.y, x.z, x.w}, {y.x, y.y, y.z, y.w}};
  uint32_t mag[2];
  gs_row_mags<true>(mag, a);
  gs_put_rows_as<true>(m, i0, j0, a, mag);
}
__device__ __forceinline__ void gs_put_rows(const GsByRow& m, int i0, int j0, const float (&a)[2][4]) {
  uint32_t mag[2];
  gs_row_mags<false>(mag, a);
  if (__any_sync(0xffffffffu, max(mag[0], mag[1]) >= kGsInf))
    gs_put_rows_odd(m, i0, j0, make_float4(a[0][0], a[0][1], a[0][2], a[0][3]), make_float4(a[1][0], a[1][1], a[1][2], a[1][3]));
  else gs_put_rows_as<false>(m, i0, j0, a, mag);
}

// ---- reading -------------------------------------------------------------------------------------------------------------------
// an element put together again, for the element-by-element products
__device__ __forceinline__ float gs_at(const GsSplit& m, int i, int l) {
  return (__half2float(m.hi[i * m.pitch + l]) + __half2float(m.lo[i * m.pitch + l])) * m.inv_s[(i >> 4) * m.sp + (l >> 4)];
}
__device__ __forceinline__ float gs_at(const GsByRow& m, int i, int l) {
  return (__half2float(m.hi[i * m.pitch + l]) + __half2float(m.lo[i * m.pitch + l])) * m.inv_s[i * m.fr + (l >> 4) * m.fc];
}
__device__ __forceinline__ void gs_add(float (&acc)[4], const float (&p)[4], float f) {
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] = fmaf(p[e], f, acc[e]);
}

}  // namespace rfa
