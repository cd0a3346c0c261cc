// fp8 (e4m3) quantisation kernels and the scaled fp8 GEMM on tcgen05 (kind::f8f6f4).
//
// The reference only emulates fp8 by rounding fp32 values (ghostflow-nn/src/mixed_precision.rs:264-285); here the
// operands are real e4m3 bytes and the product runs on the tensor cores at twice the bf16 rate.
//
// Two scaling schemes:
//   mode 0  one scale per row of A (token) and per row of B (output channel); the accumulator is scaled once in the
//           epilogue: C[m, n] = sa[m] * sb[n] * sum_k A[m, k] B[n, k].                      (128 x 256 tiles)
//   mode 1  block scales: A has one scale per row and 128-wide k block (stored [K / 128, M]), B one per 128 x 128
//           block ([N / 128, K / 128]). Every k block is accumulated in TMEM on its own and promoted into fp32
//           registers with its scale: C[m, n] = sum_kb sa[kb, m] * sb[n / 128, kb] * partial_kb.  (128 x 128 tiles)
//
// Layout of the kernel is the bf16 GEMM's: one TMA warp, one MMA warp, four epilogue warps, persistent over tiles,
// two TMEM accumulator buffers, bounded waits that record a status code and bail out.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include "gf_host.h"
#include "gf_ptx.cuh"

namespace gf {

// CTA-pair kernel (gemm2sm_bf16.cu)
int gemm2sm_wanted(int M, int N, int K);
int gemm2sm_run_fp8(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                    const float* sa, const float* sb, const void* bias, int* status, cudaStream_t stream);

constexpr int F8_BM = 128;
constexpr int F8_BK = 128;          // e4m3 elements = 128 bytes = one swizzle-128B row
constexpr int F8_THREADS = 192;
constexpr float F8_MAX = 448.f;

// ------------------------------------------------------------------ quantisation
__device__ __forceinline__ uint32_t pack_e4m3x4(float a, float b, float c, float d) {
  const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
  const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
  return lo | (hi << 16);
}

// One warp per row. mode 0: scale[row]; mode 1: scale_t[kb * T + row] per 128-wide block.
__global__ void quant_rows_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, uint8_t* __restrict__ q,
                                  long long ldq, float* __restrict__ scale, int T, int K, int mode) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= T) return;
  const __nv_bfloat16* xr = x + (long long)row * ldx;
  uint8_t* qr = q + (long long)row * ldq;
  if (mode == 0) {
    float amax = 0.f;
    for (int c = lane * 8; c < K; c += 256) {
      const uint4 u = *reinterpret_cast<const uint4*>(xr + c);
      float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), cc = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(cc.x), fabsf(cc.y)), fmaxf(fabsf(d.x), fabsf(d.y))));
    }
    for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float s = fmaxf(amax, 1e-12f) / F8_MAX;
    const float inv = 1.f / s;
    if (lane == 0) scale[row] = s;
    for (int c = lane * 8; c < K; c += 256) {
      const uint4 u = *reinterpret_cast<const uint4*>(xr + c);
      float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), cc = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
      uint2 o;
      o.x = pack_e4m3x4(a.x * inv, a.y * inv, b.x * inv, b.y * inv);
      o.y = pack_e4m3x4(cc.x * inv, cc.y * inv, d.x * inv, d.y * inv);
      *reinterpret_cast<uint2*>(qr + c) = o;
    }
  } else {
    // 16 lanes cover one 128-wide block; a warp does two blocks per step
    for (int c0 = 0; c0 < K; c0 += 256) {
      const int c = c0 + lane * 8;
      float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (c < K) {
        const uint4 u = *reinterpret_cast<const uint4*>(xr + c);
        float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), cc = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = cc.x; v[5] = cc.y; v[6] = d.x; v[7] = d.y;
      }
      float amax = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
      for (int o = 8; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
      const float s = fmaxf(amax, 1e-12f) / F8_MAX;
      const float inv = 1.f / s;
      if (c < K) {
        if ((lane & 15) == 0) scale[(long long)(c >> 7) * T + row] = s;
        uint2 o;
        o.x = pack_e4m3x4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv);
        o.y = pack_e4m3x4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv);
        *reinterpret_cast<uint2*>(qr + c) = o;
      }
    }
  }
}

// Row scales (mode 0) with the row kept in registers between the maximum and the conversion, so x is read once. TPR
// threads share a row of up to TPR * 8 * NV columns; all NV loads of a thread are issued before the first is used.
// Bound by memory (3 bytes per element); the loop above has one 16-byte load in flight per lane and reads x twice.
// [4096, 4096] and [11008, 4096] together: 43 us before, 35 us (5.3 TB/s).
template <int TPR, int NV>
__global__ void __launch_bounds__(256)
quant_rows_reg_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, uint8_t* __restrict__ q, long long ldq,
                      float* __restrict__ scale, int T, int K) {
  __shared__ float red[8];
  const int t = threadIdx.x % TPR;
  const int row = blockIdx.x * (256 / TPR) + threadIdx.x / TPR;
  const bool live = row < T;                    // rows of a CTA may end early; its barriers are for everybody
  const __nv_bfloat16* xr = x + (long long)row * ldx;
  uint4 u[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * TPR) * 8;
    u[i] = live && c < K ? *reinterpret_cast<const uint4*>(xr + c) : make_uint4(0, 0, 0, 0);
  }
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const float2 a = unpack_bf16x2(u[i].x), b = unpack_bf16x2(u[i].y), cc = unpack_bf16x2(u[i].z), d = unpack_bf16x2(u[i].w);
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(cc.x), fabsf(cc.y)), fmaxf(fabsf(d.x), fabsf(d.y))));
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if (TPR > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    const int w0 = threadIdx.x / TPR * (TPR / 32);
#pragma unroll
    for (int w = 0; w < TPR / 32; ++w) amax = fmaxf(amax, red[w0 + w]);
  }
  if (!live) return;
  const float sc = fmaxf(amax, 1e-12f) / F8_MAX;
  const float inv = 1.f / sc;
  if (t == 0) scale[row] = sc;
  uint8_t* qr = q + (long long)row * ldq;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (t + i * TPR) * 8;
    if (c < K) {
      const float2 a = unpack_bf16x2(u[i].x), b = unpack_bf16x2(u[i].y), cc = unpack_bf16x2(u[i].z), d = unpack_bf16x2(u[i].w);
      uint2 o;
      o.x = pack_e4m3x4(a.x * inv, a.y * inv, b.x * inv, b.y * inv);
      o.y = pack_e4m3x4(cc.x * inv, cc.y * inv, d.x * inv, d.y * inv);
      *reinterpret_cast<uint2*>(qr + c) = o;
    }
  }
}

// ---- quantisation along the other axis, with the transpose: x [R, C] -> qt [C, R], one scale per column of x, and
// optionally q [R, C] with one scale per row from the same two passes. The weight-gradient and input-gradient products
// contract over the rows of their stored operands, so they need x^T; writing it in bf16 first cost a strided copy per
// operand (2 + 2 bytes per element and poorly coalesced) before the quantisation read it twice.
// Pass 1 finds the maxima (order-free, so the result does not depend on the schedule), pass 2 converts a 128 x 64 tile
// and turns it in shared memory so that both outputs leave in full sectors. 5 bytes per element (6 with q), of which
// the second read mostly hits L2 for tensors below its 126 MB. dy [4096, 11008] both ways, w [11008, 4096] and
// x [4096, 4096] transposed: 541 us before, 128 us.
constexpr int QT_ROWS = 128, QT_COLS = 64, QT_AMAX_ROWS = 64, QT_AMAX_COLS = 512;

// |a| of two packed bf16 against the running maxima; a NaN operand leaves the other one, like fmaxf.
__device__ __forceinline__ uint32_t max_abs2(uint32_t m, uint32_t a) {
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&m),
                                   __habs2(*reinterpret_cast<const __nv_bfloat162*>(&a)));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// Maxima as the bits of non-negative floats, which compare like integers. row_max may be null.
__global__ void __launch_bounds__(256)
amax_rows_cols_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, unsigned* __restrict__ row_max,
                      unsigned* __restrict__ col_max, int R, int C) {
  __shared__ float part[4][QT_AMAX_COLS];
  const int cv = threadIdx.x & 63, rg = threadIdx.x >> 6;      // 64 vectors of eight columns, four row groups
  const int c = blockIdx.x * QT_AMAX_COLS + cv * 8;
  const int r0 = blockIdx.y * QT_AMAX_ROWS + rg;
  uint32_t cm[4] = {0u, 0u, 0u, 0u};
  constexpr int BATCH = 8;                       // loads issued together: the atomics below would keep them apart
  for (int i = 0; i < QT_AMAX_ROWS / 4; i += BATCH) {
    uint4 u[BATCH];
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const int r = r0 + (i + k) * 4;
      u[k] = r < R && c < C ? *reinterpret_cast<const uint4*>(x + (long long)r * ldx + c) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      const uint4 w = u[k];
      cm[0] = max_abs2(cm[0], w.x); cm[1] = max_abs2(cm[1], w.y); cm[2] = max_abs2(cm[2], w.z); cm[3] = max_abs2(cm[3], w.w);
      if (row_max) {
        const int r = r0 + (i + k) * 4;
        const float2 f = unpack_bf16x2(max_abs2(max_abs2(max_abs2(max_abs2(0u, w.x), w.y), w.z), w.w));
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(f.x, f.y)));
        if ((threadIdx.x & 31) == 0 && r < R) atomicMax(row_max + r, m);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = unpack_bf16x2(cm[j]);
    part[rg][cv * 8 + 2 * j] = f.x;
    part[rg][cv * 8 + 2 * j + 1] = f.y;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < QT_AMAX_COLS; i += 256) {
    const int cc = blockIdx.x * QT_AMAX_COLS + i;
    if (cc < C)
      atomicMax(col_max + cc, __float_as_uint(fmaxf(fmaxf(part[0][i], part[1][i]), fmaxf(part[2][i], part[3][i]))));
  }
}

// q (row-scaled [R, C]) may be null. R and C are multiples of 16.
__global__ void __launch_bounds__(256)
quant_transpose_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const float* __restrict__ row_max,
                       const float* __restrict__ col_max, uint8_t* __restrict__ q, float* __restrict__ row_scale,
                       uint8_t* __restrict__ qt, float* __restrict__ col_scale, int R, int C) {
  // [column][rows / 4] words; a pitch of 33 keeps the transposing writes two-way and the reads conflict-free
  __shared__ uint32_t tile[QT_COLS][QT_ROWS / 4 + 1];
  __shared__ float inv_c[QT_COLS], inv_r[QT_ROWS];
  const int c0 = blockIdx.x * QT_COLS, r0 = blockIdx.y * QT_ROWS;
  const int cg = threadIdx.x & 7, rg = threadIdx.x >> 3;       // this thread: columns 8 cg .. + 7, rows 4 rg .. + 3
  const int c = c0 + cg * 8, r = r0 + rg * 4;
  const bool in = r < R && c < C;                              // R % 4 == 0 and C % 8 == 0: whole patches
  uint4 u[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)
    u[k] = in ? *reinterpret_cast<const uint4*>(x + (long long)(r + k) * ldx + c) : make_uint4(0, 0, 0, 0);
  if (threadIdx.x < QT_COLS) {
    const int cc = c0 + threadIdx.x;
    if (cc < C) {
      const float sc = fmaxf(col_max[cc], 1e-12f) / F8_MAX;
      inv_c[threadIdx.x] = 1.f / sc;
      if (blockIdx.y == 0) col_scale[cc] = sc;
    }
  } else if (q && threadIdx.x < QT_COLS + QT_ROWS) {
    const int i = threadIdx.x - QT_COLS, rr = r0 + i;
    if (rr < R) {
      const float sc = fmaxf(row_max[rr], 1e-12f) / F8_MAX;
      inv_r[i] = 1.f / sc;
      if (blockIdx.x == 0) row_scale[rr] = sc;
    }
  }
  __syncthreads();
  if (in) {
    float v[4][8];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t* w = reinterpret_cast<const uint32_t*>(&u[k]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(w[j]);
        v[k][2 * j] = f.x;
        v[k][2 * j + 1] = f.y;
      }
    }
    if (q) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float s = inv_r[rg * 4 + k];
        uint2 o;
        o.x = pack_e4m3x4(v[k][0] * s, v[k][1] * s, v[k][2] * s, v[k][3] * s);
        o.y = pack_e4m3x4(v[k][4] * s, v[k][5] * s, v[k][6] * s, v[k][7] * s);
        *reinterpret_cast<uint2*>(q + (long long)(r + k) * C + c) = o;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = inv_c[cg * 8 + j];
      tile[cg * 8 + j][rg] = pack_e4m3x4(v[0][j] * s, v[1][j] * s, v[2][j] * s, v[3][j] * s);
    }
  }
  __syncthreads();
  // 64 columns x 8 pieces of 16 bytes; R % 16 == 0, so a piece is inside or outside as a whole
#pragma unroll
  for (int i = threadIdx.x; i < QT_COLS * (QT_ROWS / 16); i += 256) {
    const int col = i >> 3, piece = i & 7;
    if (c0 + col < C && r0 + piece * 16 < R) {
      const uint32_t* w = &tile[col][piece * 4];
      *reinterpret_cast<uint4*>(qt + (long long)(c0 + col) * R + r0 + piece * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// One CTA (256 threads) per 128 x 128 block of a weight [N, K]; scale [N / 128 (ceil), K / 128].
__global__ void quant_block128_kernel(const __nv_bfloat16* __restrict__ w, long long ldw, uint8_t* __restrict__ q,
                                      long long ldq, float* __restrict__ scale, int N, int K) {
  __shared__ float red[8];
  const int kb = blockIdx.x, nb = blockIdx.y;
  const int c = kb * 128 + (threadIdx.x & 15) * 8;
  const int r0 = nb * 128 + (threadIdx.x >> 4);
  float amax = 0.f;
  for (int r = r0; r < min(N, nb * 128 + 128); r += 16) {
    if (c < K) {
      const uint4 u = *reinterpret_cast<const uint4*>(w + (long long)r * ldw + c);
      float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), cc = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(cc.x), fabsf(cc.y)), fmaxf(fabsf(d.x), fabsf(d.y))));
    }
  }
  for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = 0.f;
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, red[i]);
  const float s = fmaxf(amax, 1e-12f) / F8_MAX;
  const float inv = 1.f / s;
  if (threadIdx.x == 0) scale[(long long)nb * gridDim.x + kb] = s;
  for (int r = r0; r < min(N, nb * 128 + 128); r += 16) {
    if (c < K) {
      const uint4 u = *reinterpret_cast<const uint4*>(w + (long long)r * ldw + c);
      float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), cc = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
      uint2 o;
      o.x = pack_e4m3x4(a.x * inv, a.y * inv, b.x * inv, b.y * inv);
      o.y = pack_e4m3x4(cc.x * inv, cc.y * inv, d.x * inv, d.y * inv);
      *reinterpret_cast<uint2*>(q + (long long)r * ldq + c) = o;
    }
  }
}

// ------------------------------------------------------------------ GEMM
struct F8Params {
  int M, N, K;
  __nv_bfloat16* C;
  long long ldc;
  const float* sa;          // mode 0: [M]; mode 1: [K / 128, M]
  const float* sb;          // mode 0: [N]; mode 1: [ceil(N / 128), K / 128]
  const __nv_bfloat16* bias;
  int tiles_m, tiles_n;
  int* status;
  // split-K (mode 0, skinny problems): tile index = (k slice, tile); raw partial sums are added into `ws` [M, N]
  // with vector reductions and a second kernel applies scales and bias.
  int split_k;
  float* ws;
};

// Work item -> tile and k-block range. Returns false when the slice is empty.
__device__ __forceinline__ bool f8_item(const F8Params& p, int item, int num_kb, int& tm, int& tn, int& kb0, int& nkb) {
  const int per = p.tiles_m * p.tiles_n;
  const int ks = item / per;
  const int t = item - ks * per;
  tm = t % p.tiles_m;
  tn = t / p.tiles_m;
  const int kbs = (num_kb + p.split_k - 1) / p.split_k;
  kb0 = ks * kbs;
  nkb = min(kbs, num_kb - kb0);
  return nkb > 0;
}

template <int BN>
struct F8Cfg {
  static constexpr int A_BYTES = F8_BM * F8_BK;
  static constexpr int B_BYTES = BN * F8_BK;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BN == 256) ? 4 : 6;
  static constexpr int TMEM_COLS = 2 * BN;     // 512 or 256
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

__device__ __forceinline__ void f8_set_status(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

// MODE 0: BN = 256, one drain per tile. MODE 1: BN = 128, one drain per k block.
template <int BN, int MODE>
__global__ void __launch_bounds__(F8_THREADS, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const F8Params p) {
  using Cfg = F8Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* tfull_bar = empty_bar + Cfg::STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_kb = (p.K + F8_BK - 1) / F8_BK;
  const int num_tiles = p.tiles_m * p.tiles_n * p.split_k;
  const int cta = blockIdx.x, nctas = gridDim.x;
  // accumulator hand-offs per tile: one (mode 0) or one per k block (mode 1)
  const int drains = MODE == 0 ? 1 : num_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], 4);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = cta; tile < num_tiles && ok; tile += nctas) {
        int tm, tn, kb0, nkb;
        if (!f8_item(p, tile, num_kb, tm, tn, kb0, nkb)) continue;
        for (int kb = kb0; kb < kb0 + nkb; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
            f8_set_status(p.status, GF_ERR_WAIT_EMPTY);
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          mbar_expect_tx(&full_bar[stage], Cfg::STAGE_BYTES);
          tma_load_2d(sa, &tmA, &full_bar[stage], kb * F8_BK, tm * F8_BM);
          tma_load_2d(sa + Cfg::A_BYTES, &tmB, &full_bar[stage], kb * F8_BK, tn * BN);
          if (++stage == Cfg::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_e4m3(F8_BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;      // accumulator hand-offs so far
      bool ok = true;
      for (int tile = cta; tile < num_tiles && ok; tile += nctas) {
        int tm_, tn_, kb0, nkb;
        if (!f8_item(p, tile, num_kb, tm_, tn_, kb0, nkb)) continue;
        for (int kb = kb0; kb < kb0 + nkb && ok; ++kb) {
          const bool first = MODE == 1 || kb == kb0;
          const int buf = it & 1;
          if (first) {
            if (!mbar_wait(&tempty_bar[buf], ((it >> 1) & 1) ^ 1)) {
              f8_set_status(p.status, GF_ERR_WAIT_TMEM_EMPTY);
              ok = false;
              break;
            }
            tc_fence_after();
          }
          if (!mbar_wait(&full_bar[stage], phase)) {
            f8_set_status(p.status, GF_ERR_WAIT_FULL);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t sb = sa + Cfg::A_BYTES;
          const uint32_t tmem_d = tmem_base + buf * BN;
#pragma unroll
          for (int kk = 0; kk < F8_BK / 32; ++kk) {
            const uint64_t adesc = umma_desc_sw128(sa + kk * 32, 16, 1024);
            const uint64_t bdesc = umma_desc_sw128(sb + kk * 32, 16, 1024);
            umma_f8_ss(tmem_d, adesc, bdesc, idesc, (kk > 0 || !first) ? 1u : 0u);
          }
          umma_commit(&empty_bar[stage]);
          if (++stage == Cfg::STAGES) {
            stage = 0;
            phase ^= 1;
          }
          if (MODE == 1 || kb == kb0 + nkb - 1) {
            umma_commit(&tfull_bar[buf]);
            ++it;
          }
        }
      }
    }
  } else {
    const int lane_grp = warp & 3;
    int it = 0;
    for (int tile = cta; tile < num_tiles; tile += nctas) {
      int tm, tn, kb0_, nkb_;
      if (!f8_item(p, tile, num_kb, tm, tn, kb0_, nkb_)) continue;
      const int row = tm * F8_BM + lane_grp * 32 + lane;
      const int n0 = tn * BN;
      bool ok = true;
      if constexpr (MODE == 0) {
        const int buf = it & 1;
        if (!mbar_wait_warp(&tfull_bar[buf], (it >> 1) & 1)) {
          f8_set_status(p.status, GF_ERR_WAIT_TMEM_FULL);
          break;
        }
        ++it;
        tc_fence_after();
        const float sa = row < p.M ? p.sa[row] : 0.f;
        const uint32_t taddr = tmem_base + buf * BN + ((uint32_t)(lane_grp * 32) << 16);
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(taddr + c * 32, r);
          tmem_ld_wait();
          const int col0 = n0 + c * 32;
          if (row < p.M && col0 < p.N && p.split_k > 1) {
            float* wp = p.ws + (long long)row * p.N + col0;
            if (col0 + 32 <= p.N && (p.N & 3) == 0) {
#pragma unroll
              for (int qd = 0; qd < 8; ++qd)
                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(wp + qd * 4),
                             "f"(__uint_as_float(r[qd * 4])), "f"(__uint_as_float(r[qd * 4 + 1])),
                             "f"(__uint_as_float(r[qd * 4 + 2])), "f"(__uint_as_float(r[qd * 4 + 3])) : "memory");
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.N) atomicAdd(wp + j, __uint_as_float(r[j]));
            }
          } else if (row < p.M && col0 < p.N) {
            __nv_bfloat16* cp = p.C + (long long)row * p.ldc + col0;
            if (col0 + 32 <= p.N && (p.ldc & 7) == 0) {
#pragma unroll
              for (int qd = 0; qd < 4; ++qd) {
                float v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  v[j] = __uint_as_float(r[qd * 8 + j]) * sa * __ldg(p.sb + col0 + qd * 8 + j);
                  if (p.bias) v[j] += __bfloat162float(p.bias[col0 + qd * 8 + j]);
                }
                uint4 o;
                o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
                o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
                *reinterpret_cast<uint4*>(cp + qd * 8) = o;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < p.N) {
                  float v = __uint_as_float(r[j]) * sa * p.sb[col0 + j];
                  if (p.bias) v += __bfloat162float(p.bias[col0 + j]);
                  cp[j] = __float2bfloat16(v);
                }
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[buf]);
      } else {
        float acc[BN];
#pragma unroll
        for (int j = 0; j < BN; ++j) acc[j] = 0.f;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(lane_grp * 32) << 16);
        for (int kb = 0; kb < drains; ++kb) {
          const int buf = it & 1;
          if (!mbar_wait_warp(&tfull_bar[buf], (it >> 1) & 1)) {
            f8_set_status(p.status, GF_ERR_WAIT_TMEM_FULL);
            ok = false;
            break;
          }
          ++it;
          tc_fence_after();
          const float s = (row < p.M ? __ldg(p.sa + (long long)kb * p.M + row) : 0.f) *
                          __ldg(p.sb + (long long)tn * num_kb + kb);
#pragma unroll
          for (int c = 0; c < BN / 32; ++c) {
            uint32_t r[32];
            tmem_ld32(lane_addr + buf * BN + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c * 32 + j] = fmaf(s, __uint_as_float(r[j]), acc[c * 32 + j]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty_bar[buf]);
        }
        if (!ok) break;
        if (row < p.M) {
#pragma unroll
          for (int c = 0; c < BN / 8; ++c) {
            const int col = n0 + c * 8;
            if (col >= p.N) break;
            __nv_bfloat16* cp = p.C + (long long)row * p.ldc + col;
            if (col + 8 <= p.N && (p.ldc & 7) == 0) {
              float v[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) v[j] = acc[c * 8 + j] + (p.bias ? __bfloat162float(p.bias[col + j]) : 0.f);
              uint4 o;
              o.x = pack_bf16x2(v[0], v[1]); o.y = pack_bf16x2(v[2], v[3]);
              o.z = pack_bf16x2(v[4], v[5]); o.w = pack_bf16x2(v[6], v[7]);
              *reinterpret_cast<uint4*>(cp) = o;
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (col + j < p.N)
                  cp[j] = __float2bfloat16(acc[c * 8 + j] + (p.bias ? __bfloat162float(p.bias[col + j]) : 0.f));
            }
          }
        }
      }
    }
  }

  if (p.status && *reinterpret_cast<volatile int*>(p.status) != 0) error_drain_pause();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

template <int BN, int MODE>
static int launch_f8(const CUtensorMap& tmA, const CUtensorMap& tmB, F8Params& p, cudaStream_t stream) {
  using Cfg = F8Cfg<BN>;
  static gf::DeviceOnce configured;
  auto kern = gemm_fp8_kernel<BN, MODE>;
  if (configured.todo()) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess)
      return GFH_CUDA;
    configured.mark();
  }
  p.tiles_m = (p.M + F8_BM - 1) / F8_BM;
  p.tiles_n = (p.N + BN - 1) / BN;
  int grid = sm_count();
  if (p.tiles_m * p.tiles_n * p.split_k < grid) grid = p.tiles_m * p.tiles_n * p.split_k;
  kern<<<grid, F8_THREADS, Cfg::SMEM_BYTES, stream>>>(tmA, tmB, p);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

__global__ void f8_splitk_finish_kernel(const float* __restrict__ ws, __nv_bfloat16* __restrict__ C, long long ldc,
                                        const float* __restrict__ sa, const float* __restrict__ sb,
                                        const __nv_bfloat16* __restrict__ bias, int M, int N) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)M * N) return;
  const int r = (int)(i / N), c = (int)(i % N);
  float v = ws[i] * sa[r] * sb[c];
  if (bias) v += __bfloat162float(bias[c]);
  C[(long long)r * ldc + c] = __float2bfloat16(v);
}

static float* g_f8_ws[32] = {};
static size_t g_f8_cap[32] = {};
static float* f8_workspace(size_t floats) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 32) return nullptr;
  if (g_f8_cap[dev] < floats) {
    if (g_f8_ws[dev]) cudaFree(g_f8_ws[dev]);
    size_t cap = floats < (size_t)(8 << 20) ? (size_t)(8 << 20) : floats;
    if (cudaMalloc(&g_f8_ws[dev], cap * sizeof(float)) != cudaSuccess) {
      g_f8_ws[dev] = nullptr;
      g_f8_cap[dev] = 0;
      cudaGetLastError();
      return nullptr;
    }
    g_f8_cap[dev] = cap;
  }
  return g_f8_ws[dev];
}

}  // namespace gf

using namespace gf;

// mode 0: scale [T]; mode 1: scale [K / 128, T] (K a multiple of 128).
GF_API int gf_quant_fp8_rows(const void* x, long long ldx, void* q, long long ldq, float* scale, int T, int K, int mode,
                             void* stream) {
  gf::enter();
  if (T <= 0 || K <= 0 || (K & 7) || (ldx & 7) || (ldq & 7) || (mode == 1 && (K & 127))) return GFH_BAD_ARG;
  // rows that fit in registers: 32 threads a row up to 1024 columns (no barrier needed), then the fewest threads with at
  // most eight vectors each; longer rows and block scales take the loop.
  if (mode == 0 && K <= 256 * 8 * 8) {
    const __nv_bfloat16* xb = (const __nv_bfloat16*)x;
    uint8_t* qb = (uint8_t*)q;
    cudaStream_t st = (cudaStream_t)stream;
    const int nv = K <= 1024 ? (K + 255) / 256 : K <= 4096 ? (K + 1023) / 1024 : (K + 2047) / 2048;
#define GF_QROWS(TPR, NV) \
  quant_rows_reg_kernel<TPR, NV><<<(T + 256 / TPR - 1) / (256 / TPR), 256, 0, st>>>(xb, ldx, qb, ldq, scale, T, K)
    if (K <= 1024) {
      if (nv <= 1) GF_QROWS(32, 1); else if (nv == 2) GF_QROWS(32, 2); else GF_QROWS(32, 4);
    } else if (K <= 4096) {
      if (nv <= 2) GF_QROWS(128, 2); else GF_QROWS(128, 4);
    } else {
      if (nv <= 4) GF_QROWS(256, 4); else if (nv <= 6) GF_QROWS(256, 6); else GF_QROWS(256, 8);
    }
#undef GF_QROWS
    return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
  }
  const int wpb = 8;
  quant_rows_kernel<<<(T + wpb - 1) / wpb, wpb * 32, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, ldx, (uint8_t*)q, ldq, scale, T, K, mode);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// x [R, C] bf16 (pitch ldx) -> qt [C, R] e4m3 with one scale per column of x, and, unless q is null, q [R, C] with one
// scale per row. R and C multiples of 16, x and ldx on 16-byte boundaries. scratch: fp32 [R + C].
GF_API int gf_quant_fp8_transpose(const void* x, long long ldx, void* q, float* row_scale, void* qt, float* col_scale,
                                  int R, int C, float* scratch, void* stream) {
  gf::enter();
  if (R <= 0 || C <= 0 || (R & 15) || (C & 15) || (ldx & 7) || ldx < C || !qt || !col_scale || !scratch ||
      (q && !row_scale) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(qt) & 15) ||
      (reinterpret_cast<uintptr_t>(q) & 7) || (R + QT_AMAX_ROWS - 1) / QT_AMAX_ROWS > 65535)
    return GFH_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(scratch, 0, sizeof(float) * ((size_t)R + C), st) != cudaSuccess) return GFH_CUDA;
  float* col_max = scratch;
  float* row_max = scratch + C;
  amax_rows_cols_kernel<<<dim3((C + QT_AMAX_COLS - 1) / QT_AMAX_COLS, (R + QT_AMAX_ROWS - 1) / QT_AMAX_ROWS), 256, 0, st>>>(
      (const __nv_bfloat16*)x, ldx, q ? (unsigned*)row_max : nullptr, (unsigned*)col_max, R, C);
  quant_transpose_kernel<<<dim3((C + QT_COLS - 1) / QT_COLS, (R + QT_ROWS - 1) / QT_ROWS), 256, 0, st>>>(
      (const __nv_bfloat16*)x, ldx, row_max, col_max, (uint8_t*)q, row_scale, (uint8_t*)qt, col_scale, R, C);
  gf::note_extra_launches(1);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// scale [ceil(N / 128), K / 128] (K a multiple of 128).
GF_API int gf_quant_fp8_block128(const void* w, long long ldw, void* q, long long ldq, float* scale, int N, int K,
                                 void* stream) {
  gf::enter();
  if (N <= 0 || K <= 0 || (K & 127) || (ldw & 7) || (ldq & 7)) return GFH_BAD_ARG;
  quant_block128_kernel<<<dim3(K / 128, (N + 127) / 128), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)w, ldw, (uint8_t*)q, ldq, scale, N, K);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// C[M, N] (bf16) = scaled A[M, K] (e4m3, K-major) x B[N, K]^T (e4m3, K-major); see the top of the file for `mode`.
GF_API int gf_gemm_fp8(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                       long long ldc, const float* sa, const float* sb, const void* bias, int mode, int* status,
                       void* stream_v) {
  gf::enter();
  if (M <= 0 || N <= 0 || K <= 0 || (K & 15) || (lda & 15) || (ldb & 15) || !sa || !sb) return GFH_BAD_ARG;
  if (mode == 1 && (K & 127)) return GFH_BAD_ARG;
  // large products with row and column scales run on CTA pairs (gemm2sm_bf16.cu): half the operand bytes per SM and
  // instruction, where the single-CTA tiles ask shared memory for more than it delivers. The rule is that of the bf16 products
  // (every pair has a tile of 256 x 256), but for at most 256 rows, which would leave half of a tile empty or one row of tiles,
  // and where the taller tiles leave the pairs more waves than the single CTAs have: a wave takes them 7/8 of the time.
  // [4096, 4096] x [11008, 4096]^T 162 -> 145 us, 8192^3 466 -> 392 us, [2048, 4096] x [4096, 4096]^T 40 -> 35 us. Waves of single
  // CTAs / pairs, us of each: [384, 4096] x [11008, 4096]^T 1 / 2, 23.7 / 29.5, [512, ...] 2 / 2, 35.6 / 29.9, [1040, 4096] x
  // [4096, 4096]^T 1 / 2, 23.0 / 28.5, [640, 4096] x [22016, 4096]^T 3 / 4, 56.1 / 57.2, [784, ...] 5 / 5, 76 / 70.
  const long long sms = gf::sm_count(), n_tiles = (N + 255) / 256;
  const long long waves = ((M + 127) / 128 * n_tiles + sms - 1) / sms;
  const long long pair_waves = ((M + 255) / 256 * n_tiles + sms / 2 - 1) / (sms / 2);
  if (mode == 0 && M > 256 && gf::gemm2sm_wanted(M, N, K) && 7 * pair_waves <= 8 * waves &&
      !(reinterpret_cast<uintptr_t>(sb) & 15))
    return gf::gemm2sm_run_fp8(A, B, C, M, N, K, lda, ldb, ldc, sa, sb, bias, status, (cudaStream_t)stream_v);
  const int bn = mode == 0 ? 256 : 128;
  CUtensorMap tmA, tmB;
  int rc = make_tmap_2d(&tmA, A, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, M, K, lda, F8_BM, F8_BK);
  if (rc) return rc;
  rc = make_tmap_2d(&tmB, B, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, N, K, ldb, bn, F8_BK);
  if (rc) return rc;
  F8Params p;
  p.M = M; p.N = N; p.K = K; p.C = (__nv_bfloat16*)C; p.ldc = ldc; p.sa = sa; p.sb = sb;
  p.bias = (const __nv_bfloat16*)bias; p.status = status;
  p.split_k = 1; p.ws = nullptr;
  cudaStream_t st = (cudaStream_t)stream_v;
  if (mode == 0 && M <= 256 && K >= 4096) {
    // decode-sized: split K until there is about one work item per SM (see the bf16 kernel)
    const long long tiles = (long long)((M + F8_BM - 1) / F8_BM) * ((N + 255) / 256);
    int split = (int)(sm_count() / (tiles > 0 ? tiles : 1));
    if (split > K / 1024) split = K / 1024;
    if (split > 16) split = 16;
    float* ws = split >= 2 ? f8_workspace((size_t)M * N) : nullptr;
    if (ws) {
      if (cudaMemsetAsync(ws, 0, sizeof(float) * (size_t)M * N, st) != cudaSuccess) return GFH_CUDA;
      p.split_k = split;
      p.ws = ws;
      rc = launch_f8<256, 0>(tmA, tmB, p, st);
      if (rc) return rc;
      const long long n = (long long)M * N;
      f8_splitk_finish_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(ws, (__nv_bfloat16*)C, ldc, sa, sb,
                                                                          (const __nv_bfloat16*)bias, M, N);
      gf::note_extra_launches(1);
      return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
    }
  }
  if (mode == 0) return launch_f8<256, 0>(tmA, tmB, p, st);
  if (mode == 1) return launch_f8<128, 1>(tmA, tmB, p, st);
  return GFH_BAD_ARG;
}
