// Pieces shared by the chunked kernels of the general geometries (generic_split.cu, generic_mma.cu): loads of fp16 tiles, fragments,
// products of two fp16 tiles.
#pragma once

#include <math_constants.h>

#include "common.cuh"

namespace rfa {

__host__ __device__ inline int gm_round16(int x) { return (x + 15) & ~15; }
__host__ __device__ inline int gm_groups32(int K) { return (K + 31) / 32; }

struct GmTile { const __half* p; int pitch; };

// ---- loads ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void gm_cp16(void* dst, const void* src, bool live) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void gm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void gm_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// This thread's 16-byte pieces of a tile with rows of `width` halves: the first one and the step to the next (two divisions, once a
// kernel: they were a tenth of the chunked kernels' instructions when each tile took its own)
struct GmWalk { int r, c, dr, dc, w8; };
__device__ __forceinline__ GmWalk gm_walk(int width) {
  GmWalk w;
  w.w8 = width >> 3;
  w.dr = blockDim.x / w.w8; w.dc = blockDim.x - w.dr * w.w8;
  w.r = threadIdx.x / w.w8; w.c = threadIdx.x - w.r * w.w8;
  return w;
}
// f(row, first column) of this thread's pieces of a tile of C rows
template <class F>
__device__ __forceinline__ void gm_each16(int C, const GmWalk& w, F f) {
  int r = w.r, c = w.c;
  while (r < C) {
    f(r, c * 8);
    r += w.dr;
    c += w.dc;
    if (c >= w.w8) { c -= w.w8; ++r; }
  }
}
// C rows of `width` halves, token t0 + r of sequence bh; rows from `valid` on, and masked ones, come out as zeros
__device__ __forceinline__ void gm_load(__half* dst, int pitch, const __half* src, int C, int width, const GmWalk& w, int64_t t0, int valid,
                                        int BH, int bh, const uint8_t* mrow) {
  const size_t row = (size_t)BH * width;
  src += ((size_t)t0 * BH + bh) * width;
  gm_each16(C, w, [&](int r, int c) {
    const bool live = r < valid && !(mrow && mrow[t0 + r]);
    gm_cp16(dst + r * pitch + c, src + (live ? r * row + c : 0), live);
  });
}
// has any of this thread's own chunks of the tile a non-finite value?  (after its cp.async have landed)
__device__ __forceinline__ bool gm_odd(const __half* tile, int pitch, int C, const GmWalk& walk) {
  uint32_t odd = 0;
  gm_each16(C, walk, [&](int r, int c) {
    const uint4 u = *reinterpret_cast<const uint4*>(tile + r * pitch + c);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) odd |= (w[e] & 0x7C007C00u) + 0x04000400u;      // an exponent of all ones carries into the sign's place
  });
  return (odd & 0x80008000u) != 0;
}

// ---- products --------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void gm_mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void gm_ldsm(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void gm_ldsm_t(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void gm_mma16_0(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {      // from zero
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// ldmatrix by shared-memory address: 32-bit arithmetic
__device__ __forceinline__ uint32_t gm_addr(const __half* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void gm_ldsm(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void gm_ldsm_t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
// The lane's row and column offset for the four 8 x 8 blocks of a 16 x 16 fragment: A by rows or B by rows of the inner index
// (trans) take `a`, B by rows of its columns or A by rows of the inner index (trans) take `b`.
__device__ __forceinline__ int gm_off_a(int lane, int pitch) { return (lane & 15) * pitch + (lane >> 4) * 8; }
__device__ __forceinline__ int gm_off_b(int lane, int pitch) { return ((lane & 7) + (lane >> 4) * 8) * pitch + ((lane >> 3) & 1) * 8; }
// acc (16 x 16, rows i0, columns j0) = X Y^T of two fp16 tiles stored along the inner index, `width` (rounded up to 16: zeros) long
__device__ __forceinline__ void gm_exact(float (&acc)[2][4], GmTile x, int i0, GmTile y, int j0, int width) {
  const int lane = threadIdx.x & 31;
  uint32_t pa = gm_addr(x.p + i0 * x.pitch + gm_off_a(lane, x.pitch)), pb = gm_addr(y.p + j0 * y.pitch + gm_off_b(lane, y.pitch));
#pragma unroll 4
  for (int l = 0; l < width; l += 16, pa += 32, pb += 32) {
    uint32_t a[4], b[4];
    gm_ldsm(a, pa);
    gm_ldsm(b, pb);
    float part[2][4];
    gm_mma16_0(part[0], a, b[0], b[1]);
    gm_mma16_0(part[1], a, b[2], b[3]);
#pragma unroll
    for (int e = 0; e < 4; ++e) { acc[0][e] += part[0][e]; acc[1][e] += part[1][e]; }
  }
}
// A masked product where A is triangular and B holds a non-finite value: element by element, only over the l that
// ok(i, l) admits.
template <int NT, class LA, class LB, class OK>
__device__ __noinline__ void gm_product_masked(float (&acc)[NT][4], int i0, int j0, int nt, int l0, int l1, LA la, LB lb, OK ok) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  for (int l = l0; l < l1; l += 2)
    for (int r = 0; r < 2; ++r) {
      const int i = i0 + g + 8 * r;
      const float2 a = la(i, l);
#pragma unroll
      for (int n = 0; n < NT; ++n)
        if (n < nt)
          for (int e = 0; e < 2; ++e) {
            const float2 b = lb(l, j0 + 8 * n + 2 * t + e);
            if (ok(i, l)) acc[n][2 * r + e] = fmaf(a.x, b.x, acc[n][2 * r + e]);
            if (ok(i, l + 1)) acc[n][2 * r + e] = fmaf(a.y, b.y, acc[n][2 * r + e]);
          }
    }
}
template <int NT>
__device__ __forceinline__ void gm_zero(float (&acc)[NT][4]) {
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
}
// single elements of operands
__device__ __forceinline__ float2 gm_row(GmTile x, int i, int l) {          // fp16 tile stored along l: x[i][l], x[i][l + 1]
  return __half22float2(*reinterpret_cast<const __half2*>(x.p + i * x.pitch + l));
}
__device__ __forceinline__ float2 gm_col(GmTile x, int l, int j) {          // fp16 tile stored across l: x[l][j], x[l + 1][j]
  return make_float2(__half2float(x.p[l * x.pitch + j]), __half2float(x.p[(l + 1) * x.pitch + j]));
}
__device__ __forceinline__ float2 gm_frow(const float* s, int pitch, int i, int l) { return *reinterpret_cast<const float2*>(s + i * pitch + l); }
__device__ __forceinline__ float2 gm_fcol(const float* s, int pitch, int l, int j) { return make_float2(s[l * pitch + j], s[(l + 1) * pitch + j]); }
__device__ __forceinline__ float gm_quad(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// zero the pad columns that gm_exact reads, once: the loads never touch them
__device__ __forceinline__ void gm_pad(GmTile tile, int C, int width) {
  const int w = gm_round16(width) - width;         // 0 or 8
  if (w)
    for (int i = threadIdx.x; i < C; i += blockDim.x) *reinterpret_cast<uint4*>(const_cast<__half*>(tile.p) + i * tile.pitch + width) = make_uint4(0, 0, 0, 0);
}
// qz[row] = q[row] . z, four threads per row
template <int C>
__device__ __forceinline__ void gm_qz(float* qz, GmTile q, const float* z, int K) {
  const int row = threadIdx.x >> 2;
  if (row < C) {                                       // whole warps: C is a multiple of 8
    float s = 0.f;
    for (int l = 2 * (threadIdx.x & 3); l < K; l += 8) {
      const float2 a = gm_row(q, row, l);
      s = fmaf(a.x, z[l], fmaf(a.y, z[l + 1], s));
    }
    s = gm_quad(s);
    if ((threadIdx.x & 3) == 0) qz[row] = s;
  }
}
__device__ __forceinline__ void gm_store2(__half* p, float a, float b) { *reinterpret_cast<__half2*>(p) = __floats2half2_rn(a, b); }
// inv and gz of a chunk's rows, from what sweep 1 left
__device__ __forceinline__ void gm_row_scalars(float* inv, float* gz, const float* ws_den, const float* ws_gz, int C, size_t base, int valid) {
  const int i = threadIdx.x;
  if (i < C) {
    inv[i] = i < valid ? 1.f / fmaxf(ws_den[base + i], kEps) : 0.f;
    gz[i] = i < valid ? ws_gz[base + i] : 0.f;
  }
}

}  // namespace rfa
