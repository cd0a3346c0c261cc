// bf16 GEMM for a handful of rows (one token of each sequence of a small batch):
//   C[M, N] = act(alpha * A[M, K] * W[N, K]^T + bias + residual),  M <= 16.
//
// The weight is read once and is all that counts, so the kernel is built around the load path: every lane fetches W
// with 16-byte loads straight into the A fragments of mma.m16n8k16 (16 output features), with the few rows of
// A as the B fragments (8 tokens). The contraction order is free as long as both operands use the same one: lane
// (r = lane / 4, c = lane % 4) holds k = 8c .. 8c + 7 of every 32, so one 16-byte vector of a row serves two k steps and a
// warp reads whole 128-byte lines. The warps of a CTA split K and add their sums through shared memory in a fixed
// order: no workspace to clear, no atomics, no second kernel (the tcgen05 path splits K over CTAs for such
// shapes and needs all three, and its 128-row tiles are 90 % padding). tcgen05 has nothing to offer at 8 flops a byte.
// Two 8-token tiles at most: with four, [32, 4096] x [22016, 4096]^T takes 68 us against 62 us on the tcgen05 path, because
// the rows of A are re-read from L2 by every CTA. Blocks in flight: two with one tile, one with two, where more
// registers would cost the occupancy that keeps loads in flight (49 against 59 us at [16, 4096] x [22016, 4096]^T).
// The four products of one LLaMA-7B layer (404 MB of weights), eight rows: 124 us before, 99 us (4.1 TB/s).
// Single products by events with a cold L2, before -> now: [8, 4096] x [22016, 4096]^T 64 -> 49 us, x [4096, 4096]^T
// 27 -> 18 us; [16, 4096] x [22016, 4096]^T 62 -> 49 us; [8, 11008] x [4096, 11008]^T 36 -> 33 us.
#include "gf_host.h"
#include "gf_ptx.cuh"

namespace gf {

constexpr int SK_WARPS = 8;

__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {   // read once: keep it out of L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// NT tiles of eight tokens, U k blocks of 64 in flight per warp
template <int NT, int U>
__global__ void __launch_bounds__(SK_WARPS * 32)
gemm_skinny_kernel(const __nv_bfloat16* __restrict__ A, long long lda, const __nv_bfloat16* __restrict__ W, long long ldw,
                   void* __restrict__ C, long long ldc, int out_fp32, int M, int N, int K,
                   const __nv_bfloat16* __restrict__ bias, const __nv_bfloat16* __restrict__ residual, long long ldr,
                   float alpha, int relu) {
  __shared__ float part[SK_WARPS][NT * 8][17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane >> 2, c = lane & 3;
  const int n0 = blockIdx.x * 16;
  // features past N repeat the last one and are dropped at the end; tokens past M are zero
  const __nv_bfloat16* w[2];
#pragma unroll
  for (int f = 0; f < 2; ++f) w[f] = W + (long long)min(n0 + f * 8 + r, N - 1) * ldw + 8 * c;
  const __nv_bfloat16* a[NT];
  bool live[NT];
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    live[t] = t * 8 + r < M;
    a[t] = A + (long long)(live[t] ? t * 8 + r : 0) * lda + 8 * c;
  }
  float acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;

  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (int k0 = warp * 64 * U; k0 < K; k0 += SK_WARPS * 64 * U) {
    uint4 u[U * 2][2], x[U * 2][NT];
#pragma unroll
    for (int h = 0; h < U * 2; ++h) {
      const int k = k0 + h * 32;
      const bool in = k + 8 * c < K;            // K is a multiple of eight: a vector is inside or outside as a whole
#pragma unroll
      for (int f = 0; f < 2; ++f) u[h][f] = in ? ld_stream(w[f] + k) : zero;
#pragma unroll
      for (int t = 0; t < NT; ++t) x[h][t] = in && live[t] ? __ldg(reinterpret_cast<const uint4*>(a[t] + k)) : zero;
    }
#pragma unroll
    for (int h = 0; h < U * 2; ++h)
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        mma_bf16_16816(acc[t], u[h][0].x, u[h][1].x, u[h][0].y, u[h][1].y, x[h][t].x, x[h][t].y);
        mma_bf16_16816(acc[t], u[h][0].z, u[h][1].z, u[h][0].w, u[h][1].w, x[h][t].z, x[h][t].w);
      }
  }
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    part[warp][t * 8 + 2 * c][r] = acc[t][0];
    part[warp][t * 8 + 2 * c + 1][r] = acc[t][1];
    part[warp][t * 8 + 2 * c][r + 8] = acc[t][2];
    part[warp][t * 8 + 2 * c + 1][r + 8] = acc[t][3];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < NT * 8 * 16; i += SK_WARPS * 32) {
    const int m = i >> 4, f = i & 15, n = n0 + f;
    if (m >= M || n >= N) continue;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < SK_WARPS; ++q) v += part[q][m][f];
    v *= alpha;
    if (bias) v += __bfloat162float(bias[n]);
    if (residual) v += __bfloat162float(residual[(long long)m * ldr + n]);
    if (relu) v = fmaxf(v, 0.f);
    if (out_fp32) reinterpret_cast<float*>(C)[(long long)m * ldc + n] = v;
    else reinterpret_cast<__nv_bfloat16*>(C)[(long long)m * ldc + n] = __float2bfloat16(v);
  }
}

// At most 16 rows, both operands K-major, rows on 16-byte boundaries, whole 16-byte vectors along K.
bool gemm_skinny_takes(const void* A, const void* W, int M, int N, int K, int a_mn_major, long long lda, int b_mn_major,
                       long long ldb, int accumulate) {
  return M <= 16 && !a_mn_major && !b_mn_major && !accumulate && K % 8 == 0 && lda % 8 == 0 && ldb % 8 == 0 &&
         ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0 && M > 0 && N > 0 && K > 0;
}

int gemm_skinny_run(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                    int out_fp32, const void* bias, const void* residual, long long ldr, float alpha, int relu,
                    cudaStream_t st) {
  const __nv_bfloat16 *a = (const __nv_bfloat16*)A, *w = (const __nv_bfloat16*)W;
  const __nv_bfloat16 *b = (const __nv_bfloat16*)bias, *res = (const __nv_bfloat16*)residual;
  if (M <= 8)
    gemm_skinny_kernel<1, 2><<<(N + 15) / 16, SK_WARPS * 32, 0, st>>>(a, lda, w, ldb, C, ldc, out_fp32, M, N, K, b, res,
                                                                        ldr, alpha, relu);
  else
    gemm_skinny_kernel<2, 1><<<(N + 15) / 16, SK_WARPS * 32, 0, st>>>(a, lda, w, ldb, C, ldc, out_fp32, M, N, K, b, res,
                                                                        ldr, alpha, relu);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

}  // namespace gf
