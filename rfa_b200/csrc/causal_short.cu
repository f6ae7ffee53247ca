// Causal RFA of sequences no longer than kShortMax tokens (K = 128, d = 64, no state carried in or out): forward in one
// kernel, backward from the forward's saved output in one.
//
// Such a sequence is a single chunk, so that nothing of the scan is left: no state, no products with it, no export.  What
// bounds the tcgen05 kernels here is a CTA's fixed cost -- 512 columns of tensor memory and 200 KB of shared memory admit
// one CTA per SM, whose barriers, allocation and first loads overlap nothing -- and work on 128 rows whatever the length:
// 1536 sequences of 45 tokens took 51 + 57 + 71 us for 150 MB.  Here a CTA has one warp per 16 tokens and shared memory for the
// rows there are, several fit an SM and hide each other's loads; products are mma.sync m16n8k16 on fragments from
// ldmatrix, and the score rows of a warp go from accumulators to operands without leaving its registers.  Operands
// and roundings are those of the tcgen05 kernels: fp16 P, dA and g / den, fp32 sums.
//
//   forward    P = tril(Q K^T);  raw = rowsum(P);  out = P V / max(raw, 1)
//   backward   inv = 1 / max(raw, 1);  gs = inv g;  gz = -inv (g . out) [raw > 1];  D = tril(gs V^T + gz)
//              gq = D K;   gk = D^T Q;   gv = P^T gs          (rfa.py:57-64, 79-101)
// The backward reads each input once and writes each gradient once (two sweeps read q, k, v, g twice).
#include "common.cuh"
#include "sm100.cuh"

namespace rfa {

constexpr int kShortMax = 128;
constexpr int kShPX = kK + 8, kShPY = kD + 8;      // row pitches in halves: 8 rows start in 8 different 16-byte banks

__device__ __forceinline__ uint32_t sh_addr(const __half* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void sh_ldsm(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sh_addr(p)) : "memory");
}
__device__ __forceinline__ void sh_ldsm_t(uint32_t (&r)[4], const __half* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sh_addr(p)) : "memory");
}
__device__ __forceinline__ void sh_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The four 8 x 8 blocks of a fragment load, as the lane's row and column offsets into the tile:
//   A [16 m][16 k] stored by rows m          : row lane % 16, col 8 (lane / 16)
//   B [16 k][16 n] stored by rows k (trans)  : the same
//   B stored by rows n                       : row lane % 8 + 8 (lane / 16), col 8 (lane / 8 % 2)
//   A stored by rows k (trans)               : the same
__device__ __forceinline__ int sh_off_a(int lane, int pitch) { return (lane & 15) * pitch + (lane >> 4) * 8; }
__device__ __forceinline__ int sh_off_b(int lane, int pitch) { return ((lane & 7) + (lane >> 4) * 8) * pitch + ((lane >> 3) & 1) * 8; }
__device__ __forceinline__ uint32_t sh_pack(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// R rows of `width` halves (token r of sequence bh), zeros from T on
__device__ __forceinline__ void sh_load(__half* dst, int pitch, const __half* __restrict__ src, int R, int width, int T, int BH, int bh) {
  const int w8 = width >> 3;
  for (int i = threadIdx.x; i < R * w8; i += blockDim.x) {
    const int r = i / w8, c = i % w8;
    const bool live = r < T;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sh_addr(dst + r * pitch + c * 8)),
                 "l"(src + (live ? ((size_t)r * BH + bh) * width + c * 8 : 0)), "r"(live ? 16 : 0) : "memory");
  }
}
// 16 rows of a warp's own tile from shared memory to rows i0.. of dst, 16 bytes a lane
template <int WIDTH>
__device__ __forceinline__ void sh_store(__half* __restrict__ dst, const __half* tile, int pitch, int i0, int T, int BH, int bh, int lane) {
  constexpr int w8 = WIDTH / 8;
#pragma unroll
  for (int i = lane; i < 16 * w8; i += 32) {
    const int r = i / w8, c = i % w8;
    if (i0 + r < T) *reinterpret_cast<uint4*>(dst + ((size_t)(i0 + r) * BH + bh) * WIDTH + c * 8) = *reinterpret_cast<const uint4*>(tile + r * pitch + c * 8);
  }
}
// fragment accumulators of 16 rows x 8 N columns -> fp16 rows in shared memory
template <int N>
__device__ __forceinline__ void sh_put(__half* tile, int pitch, const float (&acc)[N][4], int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int n = 0; n < N; ++n) {
    *reinterpret_cast<uint32_t*>(tile + g * pitch + n * 8 + 2 * t) = sh_pack(acc[n][0], acc[n][1]);
    *reinterpret_cast<uint32_t*>(tile + (g + 8) * pitch + n * 8 + 2 * t) = sh_pack(acc[n][2], acc[n][3]);
  }
}
// 16 x 16 block: acc += A (NK fragments of 16 k) B^T with B stored by rows n at `b` (the block's first row)
template <int NK>
__device__ __forceinline__ void sh_block(float (&acc)[2][4], const uint32_t (&a)[NK][4], const __half* b, int off) {
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;
#pragma unroll
  for (int kk = 0; kk < NK; ++kk) {
    uint32_t f[4];
    sh_ldsm(f, b + off + kk * 16);
    sh_mma(acc[0], a[kk], f[0], f[1]);
    sh_mma(acc[1], a[kk], f[2], f[3]);
  }
}
// acc (16 x 8 N) += A (one fragment of 16 k) B with B stored by rows k at `b`
template <int N>
__device__ __forceinline__ void sh_axpy(float (&acc)[N][4], const uint32_t (&a)[4], const __half* b, int off) {
#pragma unroll
  for (int n = 0; n < N; n += 2) {
    uint32_t f[4];
    sh_ldsm_t(f, b + off + n * 8);
    sh_mma(acc[n], a, f[0], f[1]);
    sh_mma(acc[n + 1], a, f[2], f[3]);
  }
}
__device__ __forceinline__ float sh_quad(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

__host__ __device__ inline uint32_t sh_fwd_bytes(int R) { return (uint32_t)R * (2 * kShPX + kShPY) * 2; }
__host__ __device__ inline uint32_t sh_bwd_bytes(int R) { return (uint32_t)R * (2 * kShPX + 2 * kShPY + 2 * (R + 8)) * 2; }

// grid (BH), one warp per 16 tokens
__global__ void __launch_bounds__(256)
causal_short_fwd_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, __half* __restrict__ out,
                        float* __restrict__ den_out, int T, int BH) {
  extern __shared__ __align__(16) __half sh_raw[];
  const int R = blockDim.x >> 1, bh = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, i0 = warp * 16;
  __half *tq = sh_raw, *tk = tq + R * kShPX, *tv = tk + R * kShPX;
  sm100::pdl_wait();
  sm100::pdl_launch_dependents();
  sh_load(tq, kShPX, q, R, kK, T, BH, bh);
  sh_load(tk, kShPX, k, R, kK, T, BH, bh);
  sh_load(tv, kShPY, v, R, kD, T, BH, bh);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  uint32_t qa[8][4];
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) sh_ldsm(qa[kk], tq + i0 * kShPX + sh_off_a(lane, kShPX) + kk * 16);
  float acc[8][4] = {}, r0 = 0.f, r1 = 0.f;
  for (int j = 0; j <= warp; ++j) {
    float s[2][4];
    sh_block<8>(s, qa, tk + j * 16 * kShPX, sh_off_b(lane, kShPX));
    if (j == warp)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (8 * n + 2 * t + (e & 1) > g + 8 * (e >> 1)) s[n][e] = 0.f;
    r0 += (s[0][0] + s[0][1]) + (s[1][0] + s[1][1]);
    r1 += (s[0][2] + s[0][3]) + (s[1][2] + s[1][3]);
    const uint32_t p[4] = {sh_pack(s[0][0], s[0][1]), sh_pack(s[0][2], s[0][3]), sh_pack(s[1][0], s[1][1]), sh_pack(s[1][2], s[1][3])};
    sh_axpy<8>(acc, p, tv + j * 16 * kShPY, sh_off_a(lane, kShPY));
  }
  r0 = sh_quad(r0); r1 = sh_quad(r1);
  if (den_out && t == 0) {
    if (i0 + g < T) den_out[(size_t)bh * T + i0 + g] = r0;
    if (i0 + g + 8 < T) den_out[(size_t)bh * T + i0 + g + 8] = r1;
  }
  const float v0 = 1.f / fmaxf(r0, kEps), v1 = 1.f / fmaxf(r1, kEps);
#pragma unroll
  for (int n = 0; n < 8; ++n) { acc[n][0] *= v0; acc[n][1] *= v0; acc[n][2] *= v1; acc[n][3] *= v1; }
  __half* mine = tq + i0 * kShPX;      // this warp's rows of Q: nobody else reads them
  __syncwarp();
  sh_put<8>(mine, kShPX, acc, lane);
  __syncwarp();
  sh_store<kD>(out, mine, kShPX, i0, T, BH, bh, lane);
}

__global__ void __launch_bounds__(256)
causal_short_bwd_kernel(const __half* __restrict__ q, const __half* __restrict__ k, const __half* __restrict__ v, const __half* __restrict__ gr,
                        const __half* __restrict__ out, const float* __restrict__ den, __half* __restrict__ gq, __half* __restrict__ gk,
                        __half* __restrict__ gv, int T, int BH) {
  extern __shared__ __align__(16) __half sh_raw[];
  const int R = blockDim.x >> 1, nw = blockDim.x >> 5, bh = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2,
            t = lane & 3, i0 = warp * 16, pp = R + 8;
  __half *tq = sh_raw, *tk = tq + R * kShPX, *tv = tk + R * kShPX, *tg = tv + R * kShPY, *tp = tg + R * kShPY, *td = tp + R * pp;
  sm100::pdl_wait();
  sm100::pdl_launch_dependents();
  sh_load(tg, kShPY, gr, R, kD, T, BH, bh);
  sh_load(tv, kShPY, v, R, kD, T, BH, bh);
  sh_load(tq, kShPX, q, R, kK, T, BH, bh);
  sh_load(tk, kShPX, k, R, kK, T, BH, bh);
  // two lanes per row of this warp: half a row of the saved output each
  const int r = lane >> 1, half = (lane & 1) * 32;
  uint4 o[4];
  float raw = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c) o[c] = make_uint4(0, 0, 0, 0);
  if (i0 + r < T) {
    const uint4* src = reinterpret_cast<const uint4*>(out + ((size_t)(i0 + r) * BH + bh) * kD + half);
#pragma unroll
    for (int c = 0; c < 4; ++c) o[c] = src[c];
    raw = den[(size_t)bh * T + i0 + r];
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  // gs = g / den over g, gz
  float gz;
  {
    const float inv = 1.f / fmaxf(raw, kEps);
    __half* row = tg + (i0 + r) * kShPY + half;
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float a[8], b[8];
      load8(row + c * 8, a);
      load8(reinterpret_cast<const __half*>(&o[c]), b);
#pragma unroll
      for (int e = 0; e < 8; ++e) { dot = fmaf(a[e], b[e], dot); a[e] *= inv; }
      store8(row + c * 8, a);
    }
    dot += __shfl_xor_sync(0xffffffffu, dot, 1);
    gz = raw > kEps ? -dot * inv : 0.f;                            // strict >, upstream rfa.py:91
  }
  const float z0 = __shfl_sync(0xffffffffu, gz, 2 * g), z1 = __shfl_sync(0xffffffffu, gz, 2 * (g + 8));
  __syncwarp();
  float aq[16][4] = {};
  {
    uint32_t qa[8][4], ga[4][4];
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) sh_ldsm(qa[kk], tq + i0 * kShPX + sh_off_a(lane, kShPX) + kk * 16);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) sh_ldsm(ga[kk], tg + i0 * kShPY + sh_off_a(lane, kShPY) + kk * 16);
    for (int j = 0; j <= warp; ++j) {
      float s[2][4], d[2][4];
      sh_block<8>(s, qa, tk + j * 16 * kShPX, sh_off_b(lane, kShPX));
      sh_block<4>(d, ga, tv + j * 16 * kShPY, sh_off_b(lane, kShPY));
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          d[n][e] += e < 2 ? z0 : z1;
          if (j == warp && 8 * n + 2 * t + (e & 1) > g + 8 * (e >> 1)) s[n][e] = d[n][e] = 0.f;
        }
      sh_put<2>(tp + i0 * pp + j * 16, pp, s, lane);
      sh_put<2>(td + i0 * pp + j * 16, pp, d, lane);
      const uint32_t a[4] = {sh_pack(d[0][0], d[0][1]), sh_pack(d[0][2], d[0][3]), sh_pack(d[1][0], d[1][1]), sh_pack(d[1][2], d[1][3])};
      sh_axpy<16>(aq, a, tk + j * 16 * kShPX, sh_off_a(lane, kShPX));
    }
  }
  __syncthreads();                               // P, D and gs are complete; K and V have been read
  __half *mk = tk + i0 * kShPX, *mv = tv + i0 * kShPY;      // this warp's rows of K and V: staging from here on
  sh_put<16>(mk, kShPX, aq, lane);
  __syncwarp();
  sh_store<kK>(gq, mk, kShPX, i0, T, BH, bh, lane);
  float ak[16][4] = {}, av[8][4] = {};
  for (int j = warp; j < nw; ++j) {              // queries from this warp's keys on
    uint32_t a[4];
    sh_ldsm_t(a, tp + j * 16 * pp + i0 + sh_off_b(lane, pp));
    sh_axpy<8>(av, a, tg + j * 16 * kShPY, sh_off_a(lane, kShPY));
    sh_ldsm_t(a, td + j * 16 * pp + i0 + sh_off_b(lane, pp));
    sh_axpy<16>(ak, a, tq + j * 16 * kShPX, sh_off_a(lane, kShPX));
  }
  __syncwarp();
  sh_put<16>(mk, kShPX, ak, lane);
  sh_put<8>(mv, kShPY, av, lane);
  __syncwarp();
  sh_store<kK>(gk, mk, kShPX, i0, T, BH, bh, lane);
  sh_store<kD>(gv, mv, kShPY, i0, T, BH, bh, lane);
}

int causal_short_max() { return kShortMax; }

static int sh_reserve(const void* kernel, uint32_t smem, const char* what) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e == cudaSuccess ? 0 : fail((int)e, "%s: cannot reserve %u bytes of shared memory: %s", what, smem, cudaGetErrorString(e));
}
int launch_causal_short_fwd(const __half* q, const __half* k, const __half* v, __half* out, float* den_out, int64_t T, int BH, cudaStream_t st) {
  const int warps = (int)(T + 15) / 16;
  const uint32_t smem = sh_fwd_bytes(warps * 16);
  if (int e = sh_reserve((const void*)causal_short_fwd_kernel, sh_fwd_bytes(kShortMax), "causal_fwd")) return e;
  sm100::launch_pdl(causal_short_fwd_kernel, dim3(BH), dim3(warps * 32), smem, st, q, k, v, out, den_out, (int)T, BH);
  return check_launch("rfa_causal_fwd (short)");
}
int launch_causal_short_bwd(const __half* q, const __half* k, const __half* v, const __half* g, const __half* out, const float* den, __half* gq,
                            __half* gk, __half* gv, int64_t T, int BH, cudaStream_t st) {
  const int warps = (int)(T + 15) / 16;
  const uint32_t smem = sh_bwd_bytes(warps * 16);
  if (int e = sh_reserve((const void*)causal_short_bwd_kernel, sh_bwd_bytes(kShortMax), "causal_bwd")) return e;
  sm100::launch_pdl(causal_short_bwd_kernel, dim3(BH), dim3(warps * 32), smem, st, q, k, v, g, out, den, gq, gk, gv, (int)T, BH);
  return check_launch("rfa_causal_bwd_saved (short)");
}

}  // namespace rfa
