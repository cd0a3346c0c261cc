// RMSNorm and LayerNorm, forward and backward, bf16 in/out with fp32 arithmetic.
//
// Bound by memory: every tensor is read once and written once, as 16-byte vectors that stay packed in registers between
// the passes over a row. Rows up to 1024 columns belong to one warp (sums are shuffles, eight rows to a CTA) if there are
// enough of them, all others to one CTA of 256 threads with one barrier per reduction. The weight / bias gradients are cross-row sums: every CTA of a
// grid that fits the machine at once keeps them in registers over its rows, with the next row's loads in flight
// behind the reduction of the current one, and writes one partial row to a scratch buffer; a second small kernel folds
// the partial rows.
//
// Measured, before -> now: RMSNorm with residual of [8192, 4096] forward 58 -> 40 us, backward 70 -> 56 us (fold included);
// LayerNorm of [8192, 768] forward 12.4 -> 7.6 us, backward 47 -> 16 us, of [8192, 8192] (one CTA to an SM, no prefetch) backward
// 264 -> 137 us, of [16, 8192] 15.8 -> 8.9 us; four column sums of a GPT-2 block 56 -> 36 us. The
// forward pass read h back from memory right after storing it (to normalise what was stored); the backward pass had
// 592 CTAs on 444 places, two barriers a row and, for short rows, eight warps adding into shared memory with atomics.
//
// Formulas follow the reference's CPU code: RMSNorm x / sqrt(mean(x^2) + eps) * w
// (ghostflow-nn/src/llama.rs:154-185); LayerNorm with biased variance
// (ghostflow-nn/src/norm.rs:239-270). The reference only names GPU kernels for these
// (ghostflow-cuda/src/kernels/mod.rs:103-106) without implementing them.
#include "gf_host.h"
#include "gf_ptx.cuh"

namespace gf {

constexpr int NORM_THREADS = 256;
constexpr int NORM_WARPS = NORM_THREADS / 32;
constexpr int NORM_MAXV = 4;      // 16-byte vectors per thread kept in registers -> D <= 8192
constexpr int NORM_WARP_D = 1024; // longest row of the one-warp kernels

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sum over the CTA with one barrier; `red` holds a float per warp and must not be written again before every thread has
// passed another barrier (callers alternate between two).
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < NORM_WARPS; ++i) t += red[i];
  return t;
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]); u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]); u.w = pack_bf16x2(f[6], f[7]);
  return u;
}
__device__ __forceinline__ uint4 ldv(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void stv(__nv_bfloat16* p, const uint4& u) { *reinterpret_cast<uint4*>(p) = u; }

struct NormFwd {
  const __nv_bfloat16 *x, *res, *w, *b;   // res: RMSNorm with the residual add in front, h = x + res
  __nv_bfloat16 *y, *h;
  float *mean, *rstd;
  int T, D;
  float eps;
};

// ------------------------------------------------------------------ forward
// One row: NV vectors of this thread at v0, v0 + stride, ...; SUM adds over all threads of the row.
template <bool LN, int NV, typename Sum>
__device__ __forceinline__ void norm_fwd_row(const NormFwd& p, int row, int v0, int stride, bool first, Sum sum) {
  const int nv = p.D >> 3;
  const long long base = (long long)row * p.D;
  uint4 xp[NV], rp[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = v0 + i * stride;
    xp[i] = v < nv ? ldv(p.x + base + v * 8) : make_uint4(0, 0, 0, 0);
    if (!LN && p.res) rp[i] = v < nv ? ldv(p.res + base + v * 8) : make_uint4(0, 0, 0, 0);
  }
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = v0 + i * stride;
    float f[8];
    unpack8(xp[i], f);
    if (!LN && p.res) {
      float r[8];
      unpack8(rp[i], r);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += r[j];
      if (p.h) {
        // normalise exactly what is stored (bf16-rounded) so backward sees the same h
        xp[i] = pack8(f);
        if (v < nv) stv(p.h + base + v * 8, xp[i]);
        unpack8(xp[i], f);
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += LN ? f[j] : f[j] * f[j];
  }
  float mean = 0.f, rstd;
  s = sum(s);
  if (LN) {
    mean = s / (float)p.D;
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (v0 + i * stride < nv) {
        float f[8];
        unpack8(xp[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) sq += (f[j] - mean) * (f[j] - mean);
      }
    }
    rstd = rsqrtf(sum(sq) / (float)p.D + p.eps);
  } else {
    rstd = rsqrtf(s / (float)p.D + p.eps);
  }
  if (first) {
    if (LN && p.mean) p.mean[row] = mean;
    if (p.rstd) p.rstd[row] = rstd;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = v0 + i * stride;
    if (v < nv) {
      float f[8], wv[8], bv[8], o[8];
      unpack8(xp[i], f);
      unpack8(ldv(p.w + v * 8), wv);
      if (!LN && p.res && !p.h) {         // the sum was not stored: it is normalised unrounded
        float r[8];
        unpack8(rp[i], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += r[j];
      }
      if (LN && p.b) unpack8(ldv(p.b + v * 8), bv);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        o[j] = LN ? (f[j] - mean) * rstd * wv[j] + (p.b ? bv[j] : 0.f) : f[j] * rstd * wv[j];
      stv(p.y + base + v * 8, pack8(o));
    }
  }
}

template <bool LN, int NV>
__global__ void __launch_bounds__(NORM_THREADS) norm_fwd_warp_kernel(const NormFwd p) {
  const int row = blockIdx.x * NORM_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row < p.T) norm_fwd_row<LN, NV>(p, row, lane, 32, lane == 0, [](float v) { return warp_sum(v); });
}

template <bool LN, int NV>
__global__ void __launch_bounds__(NORM_THREADS) norm_fwd_block_kernel(const NormFwd p) {
  __shared__ float red[2][NORM_WARPS];
  int k = 0;
  norm_fwd_row<LN, NV>(p, blockIdx.x, threadIdx.x, NORM_THREADS, threadIdx.x == 0,
                       [&](float v) { return block_sum(v, red[k++ & 1]); });
}

// ------------------------------------------------------------------ backward
// RMSNorm:   dx = rstd * g - x * rstd^3 * mean(g * x), g = dy * w ; dw = sum_rows dy * x * rstd
// LayerNorm: xhat = (x - mean) * rstd ; dx = rstd * (g - mean(g) - xhat * mean(g * xhat)) ; dw = sum dy * xhat, db = sum dy
// If `dres` is given, it is added into dx (gradient arriving through the residual branch).
struct NormBwd {
  const __nv_bfloat16 *x, *w, *dy, *dres;
  const float *mean, *rstd;
  __nv_bfloat16 *dx, *dx2;            // dx2: a second copy, for an input whose gradient is stored apart (may be null)
  float *dw_partial, *db_partial;     // one row of D per CTA
  int T, D;
};

// RES: there may be a dres. RMSNorm loads it with the row; LayerNorm, which has no registers left for that, where it is added,
// and it has kernels without. TWO: dx2 is written, which no other call pays for ([8192, 1024] 16.2 us, 17.3 with a test in the loop).
template <int NV, bool EARLY>
struct NormBwdRow {
  uint4 x[NV], g[NV], r[EARLY ? NV : 1];
  float mean, rstd;
};

template <bool LN, int NV>
__device__ __forceinline__ void norm_bwd_load(const NormBwd& p, NormBwdRow<NV, !LN>& t, int row, int v0, int stride) {
  const int nv = p.D >> 3;
  const long long base = (long long)row * p.D;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = v0 + i * stride;
    const bool in = v < nv;
    t.x[i] = in ? ldv(p.x + base + v * 8) : make_uint4(0, 0, 0, 0);
    t.g[i] = in ? ldv(p.dy + base + v * 8) : make_uint4(0, 0, 0, 0);
    if (!LN && p.dres) t.r[LN ? 0 : i] = in ? ldv(p.dres + base + v * 8) : make_uint4(0, 0, 0, 0);
  }
  t.rstd = p.rstd[row];
  t.mean = LN ? p.mean[row] : 0.f;
}

// Rows row0, row0 + step, ... of one warp or CTA; the sums over rows end in dw / db. wv: this thread's weights, packed.
template <bool LN, int NV, bool RES, bool TWO, bool PREFETCH, typename Sum>
__device__ __forceinline__ void norm_bwd_rows(const NormBwd& p, int row0, int step, int v0, int stride, float (&dw)[NV][8],
                                              float (&db)[LN ? NV : 1][8], Sum sum) {
  const int nv = p.D >> 3;
  const float inv_d = 1.f / (float)p.D;
  NormBwdRow<NV, !LN> cur, nxt;
  if (PREFETCH && row0 < p.T) norm_bwd_load<LN, NV>(p, cur, row0, v0, stride);
  for (int row = row0; row < p.T; row += step) {
    if (!PREFETCH) norm_bwd_load<LN, NV>(p, cur, row, v0, stride);
    else if (row + step < p.T) norm_bwd_load<LN, NV>(p, nxt, row + step, v0, stride);
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if (v0 + i * stride < nv) {
        float xv[8], gv[8], wv[8];
        unpack8(cur.x[i], xv); unpack8(cur.g[i], gv); unpack8(ldv(p.w + (v0 + i * stride) * 8), wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (LN) {
            const float xh = (xv[j] - cur.mean) * cur.rstd, g = gv[j] * wv[j];
            dw[i][j] += gv[j] * xh;
            db[i][j] += gv[j];
            s1 += g;
            s2 += g * xh;
          } else {
            dw[i][j] += gv[j] * xv[j] * cur.rstd;
            s2 += gv[j] * wv[j] * xv[j];
          }
        }
      }
    }
    if (LN) s1 = sum(s1) * inv_d;
    s2 = sum(s2);
    const float c = LN ? s2 * inv_d : s2 * cur.rstd * cur.rstd * cur.rstd * inv_d;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = v0 + i * stride;
      if (v < nv) {
        float xv[8], gv[8], wv[8], o[8];
        unpack8(cur.x[i], xv); unpack8(cur.g[i], gv); unpack8(ldv(p.w + v * 8), wv);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          o[j] = LN ? cur.rstd * (gv[j] * wv[j] - s1 - (xv[j] - cur.mean) * cur.rstd * c)
                    : cur.rstd * gv[j] * wv[j] - c * xv[j];
        if (RES && p.dres) {
          float rv[8];
          unpack8(LN ? ldv(p.dres + (long long)row * p.D + v * 8) : cur.r[LN ? 0 : i], rv);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += rv[j];
        }
        const uint4 out = pack8(o);
        stv(p.dx + (long long)row * p.D + v * 8, out);
        if (TWO) stv(p.dx2 + (long long)row * p.D + v * 8, out);
      }
    }
    if (PREFETCH) cur = nxt;
  }
}

// One warp per row, D <= 1024. The eight warps' sums meet in shared memory, warp by warp in its own row of it.
template <bool LN, int NV, bool RES, bool TWO>
__global__ void __launch_bounds__(NORM_THREADS, NV == 1 ? 3 : 2) norm_bwd_warp_kernel(const NormBwd p) {
  __shared__ float acc[NORM_WARPS][NORM_WARP_D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nv = p.D >> 3;
  float dw[NV][8], db[LN ? NV : 1][8];
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dw[i][j] = 0.f;
      if (LN) db[LN ? i : 0][j] = 0.f;
    }
  norm_bwd_rows<LN, NV, RES, TWO, NV <= 2>(p, blockIdx.x * NORM_WARPS + warp, gridDim.x * NORM_WARPS, lane, 32, dw, db,
                              [](float v) { return warp_sum(v); });
  auto flush = [&](const float(&a)[NV][8], float* out) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + i * 32;
      if (v < nv) {
        *reinterpret_cast<float4*>(&acc[warp][v * 8]) = make_float4(a[i][0], a[i][1], a[i][2], a[i][3]);
        *reinterpret_cast<float4*>(&acc[warp][v * 8 + 4]) = make_float4(a[i][4], a[i][5], a[i][6], a[i][7]);
      }
    }
    __syncthreads();
    for (int d = threadIdx.x; d < p.D; d += NORM_THREADS) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < NORM_WARPS; ++q) t += acc[q][d];
      out[(long long)blockIdx.x * p.D + d] = t;
    }
  };
  flush(dw, p.dw_partial);
  if constexpr (LN) {
    __syncthreads();
    flush(db, p.db_partial);
  }
}

// CTAs of a persistent grid per SM; the next row is prefetched where the registers for it are there.
template <bool LN, int NV>
constexpr int norm_bwd_ctas() { return NV == 1 ? 4 : NV == 2 ? 2 : LN ? 1 : 2; }

template <bool LN, int NV, bool RES, bool TWO>
__global__ void __launch_bounds__(NORM_THREADS, norm_bwd_ctas<LN, NV>()) norm_bwd_block_kernel(const NormBwd p) {
  __shared__ float red[4][NORM_WARPS];
  const int nv = p.D >> 3;
  float dw[NV][8], db[LN ? NV : 1][8];
#pragma unroll
  for (int i = 0; i < NV; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dw[i][j] = 0.f;
      if (LN) db[LN ? i : 0][j] = 0.f;
    }
  int k = 0;
  norm_bwd_rows<LN, NV, RES, TWO, NV <= 2>(p, blockIdx.x, gridDim.x, threadIdx.x, NORM_THREADS, dw, db,
                                 [&](float v) { return block_sum(v, red[k++ & 3]); });
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = threadIdx.x + i * NORM_THREADS;
    if (v < nv) {
      float* dst = p.dw_partial + (long long)blockIdx.x * p.D + v * 8;
      *reinterpret_cast<float4*>(dst) = make_float4(dw[i][0], dw[i][1], dw[i][2], dw[i][3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(dw[i][4], dw[i][5], dw[i][6], dw[i][7]);
      if (LN) {
        const float(&a)[8] = db[LN ? i : 0];
        dst = p.db_partial + (long long)blockIdx.x * p.D + v * 8;
        *reinterpret_cast<float4*>(dst) = make_float4(a[0], a[1], a[2], a[3]);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(a[4], a[5], a[6], a[7]);
      }
    }
  }
}

// Fold `nparts` partial rows of length D; writes bf16 (optionally accumulating into existing bf16). A second pair of
// buffers is folded by the CTAs with blockIdx.y = 1. One CTA per 32 columns: its warps stride over the partial rows (each
// reads 128 contiguous bytes of a row, four rows in flight), and their sums are added in shared memory. 32 warps, or eight for at
// most FOLD_FEW rows, where a CTA of 1024 threads takes longer to start than to fold (RMSNorm backward of one row of 4096 with its
// fold 4.9 us against 5.3, of 64 rows of 768 4.4 against 4.7).
constexpr int FOLD_FEW = 64;
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
fold_partials_kernel(const float* __restrict__ partial0, __nv_bfloat16* __restrict__ out0,
                     const float* __restrict__ partial1, __nv_bfloat16* __restrict__ out1, int nparts, int D,
                     int accumulate) {
  __shared__ float sm[WARPS][33];
  const float* partial = blockIdx.y ? partial1 : partial0;
  __nv_bfloat16* out = blockIdx.y ? out1 : out0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (d < D) {
#pragma unroll 4
    for (int p = warp; p < nparts; p += WARPS) s += partial[(long long)p * D + d];
  }
  sm[warp][lane] = s;
  __syncthreads();
  if constexpr (WARPS == 32) {      // warp w adds column w over the 32 sums
    const float t = warp_sum(sm[lane][warp]);
    const int c = blockIdx.x * 32 + warp;
    if (lane == 0 && c < D) out[c] = __float2bfloat16(accumulate ? t + __bfloat162float(out[c]) : t);
  } else if (warp == 0 && d < D) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) t += sm[w][lane];
    out[d] = __float2bfloat16(accumulate ? t + __bfloat162float(out[d]) : t);
  }
}

// ------------------------------------------------------------------ column sums (bias gradients)
// out[d] = sum over rows of x[row, d]. A CTA takes 256 columns (32 threads of one 16-byte vector each, eight row groups) and
// every gridDim.y-th batch of eight rows, four batches in flight, and writes one partial row; fold_partials_kernel adds them.
__global__ void __launch_bounds__(NORM_THREADS)
colsum_partial_kernel(const __nv_bfloat16* __restrict__ x, long long ld, float* __restrict__ partial, int T, int D) {
  __shared__ float acc[8][256];
  const int cv = threadIdx.x & 31, rg = threadIdx.x >> 5;
  const int c = blockIdx.x * 256 + cv * 8;
  float a[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = 0.f;
  if (c < D) {
#pragma unroll 4
    for (int row = blockIdx.y * 8 + rg; row < T; row += gridDim.y * 8) {
      float f[8];
      unpack8(ldv(x + (long long)row * ld + c), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += f[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[rg][cv * 8 + j] = a[j];
  __syncthreads();
  const int d = blockIdx.x * 256 + threadIdx.x;
  if (d < D) {
    float t = 0.f;
#pragma unroll
    for (int g = 0; g < 8; ++g) t += acc[g][threadIdx.x];
    partial[(long long)blockIdx.y * D + d] = t;
  }
}

static inline int norm_grid(int T) {
  int g = sm_count() * 4;
  return T < g ? T : g;
}
static inline int at_most(long long a, long long b) { return (int)(a < b ? a : b); }

static void launch_fold(const float* p0, void* o0, const float* p1, void* o1, int nparts, int D, int accumulate,
                        cudaStream_t st) {
  const dim3 grid((D + 31) / 32, o1 ? 2 : 1);
  if (nparts <= FOLD_FEW)
    fold_partials_kernel<8><<<grid, 256, 0, st>>>(p0, (__nv_bfloat16*)o0, p1, (__nv_bfloat16*)o1, nparts, D, accumulate);
  else
    fold_partials_kernel<32><<<grid, 1024, 0, st>>>(p0, (__nv_bfloat16*)o0, p1, (__nv_bfloat16*)o1, nparts, D, accumulate);
}

// A row to a warp, eight rows to a CTA, for rows that are short or many. Few rows of 264 columns and more (up to five for an SM
// forward, one backward) leave SMs idle that way and take a CTA each. RMSNorm with residual, us as CTAs / as warps: forward [16, 1024] 2.1 / 3.1, [600, 1024] 2.7 / 3.5, [600, 264]
// 2.6 / 2.6, [1200, 768] 3.6 / 3.1; backward [16, 1024] 4.2 / 6.1, [128, 264] 4.4 / 4.8, [300, 384] 5.6 / 5.1, [600, 1024] 7.3 / 6.9.
static inline bool norm_row_per_warp(int T, int D, int few) { return D <= NORM_WARP_D && !(D > 256 && T <= few); }

template <bool LN>
static int launch_norm_fwd(const NormFwd& p, cudaStream_t st) {
  if (norm_row_per_warp(p.T, p.D, sm_count() * 5)) {
    const int vpl = (p.D / 8 + 31) / 32, grid = (p.T + NORM_WARPS - 1) / NORM_WARPS;
    auto kern = vpl == 1 ? norm_fwd_warp_kernel<LN, 1> : vpl == 2 ? norm_fwd_warp_kernel<LN, 2>
                : vpl == 3 ? norm_fwd_warp_kernel<LN, 3> : norm_fwd_warp_kernel<LN, 4>;
    kern<<<grid, NORM_THREADS, 0, st>>>(p);
  } else {
    auto kern = p.D <= NORM_THREADS * 8 ? norm_fwd_block_kernel<LN, 1>
                : p.D <= NORM_THREADS * 16 ? norm_fwd_block_kernel<LN, 2> : norm_fwd_block_kernel<LN, NORM_MAXV>;
    kern<<<p.T, NORM_THREADS, 0, st>>>(p);
  }
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// Number of partial rows written: at most norm_grid(T), which sizes the caller's scratch, and no more CTAs than are
// resident at once (a second wave would wait for the first one's row loops).
template <bool LN, bool RES, bool TWO = false>
static int launch_norm_bwd(const NormBwd& p, cudaStream_t st) {
  const int cap = norm_grid(p.T), sms = sm_count();
  int grid;
  if (norm_row_per_warp(p.T, p.D, sms)) {
    const int vpl = (p.D / 8 + 31) / 32;
    grid = at_most(at_most((p.T + NORM_WARPS - 1) / NORM_WARPS, cap), (long long)sms * (vpl == 1 ? 3 : 2));
    auto kern = vpl == 1 ? norm_bwd_warp_kernel<LN, 1, RES, TWO> : vpl == 2 ? norm_bwd_warp_kernel<LN, 2, RES, TWO>
                : vpl == 3 ? norm_bwd_warp_kernel<LN, 3, RES, TWO> : norm_bwd_warp_kernel<LN, 4, RES, TWO>;
    kern<<<grid, NORM_THREADS, 0, st>>>(p);
  } else if (p.D <= NORM_THREADS * 8) {
    grid = at_most(cap, (long long)sms * norm_bwd_ctas<LN, 1>());
    norm_bwd_block_kernel<LN, 1, RES, TWO><<<grid, NORM_THREADS, 0, st>>>(p);
  } else if (p.D <= NORM_THREADS * 16) {
    grid = at_most(cap, (long long)sms * norm_bwd_ctas<LN, 2>());
    norm_bwd_block_kernel<LN, 2, RES, TWO><<<grid, NORM_THREADS, 0, st>>>(p);
  } else {
    grid = at_most(cap, (long long)sms * norm_bwd_ctas<LN, NORM_MAXV>());
    norm_bwd_block_kernel<LN, NORM_MAXV, RES, TWO><<<grid, NORM_THREADS, 0, st>>>(p);
  }
  return grid;
}

}  // namespace gf

using namespace gf;

GF_API int gf_norm_bwd_grid(int T) { return norm_grid(T); }

GF_API int gf_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int T,
                          int D, float eps, void* stream) {
  gf::enter();
  if (D % 8 || D > NORM_THREADS * NORM_MAXV * 8 || T <= 0) return GFH_BAD_ARG;
  NormFwd p{(const __nv_bfloat16*)x, (const __nv_bfloat16*)res, (const __nv_bfloat16*)w, nullptr, (__nv_bfloat16*)y,
            (__nv_bfloat16*)h_out, nullptr, rstd, T, D, eps};
  return launch_norm_fwd<false>(p, (cudaStream_t)stream);
}

// scratch: fp32 [gf_norm_bwd_grid(T), D]. dw is bf16 [D]; accumulate=1 adds into it.
// dx2: the input gradient once more (may be null).
GF_API int gf_rmsnorm_bwd2(const void* x, const void* w, const void* dy, const float* rstd, const void* dres, void* dx, void* dx2,
                           void* dw, float* scratch, int T, int D, int accumulate, void* stream) {
  gf::enter();
  if (D % 8 || D > NORM_THREADS * NORM_MAXV * 8 || T <= 0) return GFH_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  NormBwd p{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)dres, nullptr,
            rstd, (__nv_bfloat16*)dx, (__nv_bfloat16*)dx2, scratch, nullptr, T, D};
  const int parts = dx2 ? launch_norm_bwd<false, true, true>(p, st) : launch_norm_bwd<false, true>(p, st);
  launch_fold(scratch, dw, nullptr, nullptr, parts, D, accumulate, st);
  gf::note_extra_launches(1);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}
GF_API int gf_rmsnorm_bwd(const void* x, const void* w, const void* dy, const float* rstd, const void* dres,
                          void* dx, void* dw, float* scratch, int T, int D, int accumulate, void* stream) {
  return gf_rmsnorm_bwd2(x, w, dy, rstd, dres, dx, nullptr, dw, scratch, T, D, accumulate, stream);
}

// x: bf16 [T, D] with row pitch ld (elements, multiple of 8); out: bf16 [D]; scratch: fp32 [gf_norm_bwd_grid(T), D].
GF_API int gf_colsum_bf16(const void* x, long long ld, void* out, float* scratch, int T, int D, int accumulate,
                          void* stream) {
  gf::enter();
  if (D % 8 || ld % 8 || ld < D || D > NORM_THREADS * NORM_MAXV * 8 || T <= 0 || !scratch) return GFH_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int gx = (D + 255) / 256;
  // about four CTAs on an SM, each with at least one batch of eight rows
  const int gy = at_most(at_most((T + 7) / 8, norm_grid(T)), (sm_count() * 4 + gx - 1) / gx);
  colsum_partial_kernel<<<dim3(gx, gy), NORM_THREADS, 0, st>>>((const __nv_bfloat16*)x, ld, scratch, T, D);
  launch_fold(scratch, out, nullptr, nullptr, gy, D, accumulate, st);
  gf::note_extra_launches(1);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

GF_API int gf_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, int T,
                            int D, float eps, void* stream) {
  gf::enter();
  if (D % 8 || D > NORM_THREADS * NORM_MAXV * 8 || T <= 0) return GFH_BAD_ARG;
  NormFwd p{(const __nv_bfloat16*)x, nullptr, (const __nv_bfloat16*)w, (const __nv_bfloat16*)b, (__nv_bfloat16*)y, nullptr,
            mean, rstd, T, D, eps};
  return launch_norm_fwd<true>(p, (cudaStream_t)stream);
}

// scratch: fp32 [2, gf_norm_bwd_grid(T), D]. dres is added into dx (may be null).
GF_API int gf_layernorm_bwd_res(const void* x, const void* w, const void* dy, const float* mean, const float* rstd,
                                const void* dres, void* dx, void* dw, void* db, float* scratch, int T, int D, int accumulate,
                                void* stream) {
  gf::enter();
  if (D % 8 || D > NORM_THREADS * NORM_MAXV * 8 || T <= 0) return GFH_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  float* s2 = scratch + (long long)norm_grid(T) * D;
  NormBwd p{(const __nv_bfloat16*)x, (const __nv_bfloat16*)w, (const __nv_bfloat16*)dy, (const __nv_bfloat16*)dres, mean,
            rstd, (__nv_bfloat16*)dx, nullptr, scratch, s2, T, D};
  const int parts = dres ? launch_norm_bwd<true, true>(p, st) : launch_norm_bwd<true, false>(p, st);
  launch_fold(scratch, dw, s2, db, parts, D, accumulate, st);
  gf::note_extra_launches(1);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}
GF_API int gf_layernorm_bwd(const void* x, const void* w, const void* dy, const float* mean, const float* rstd,
                            void* dx, void* dw, void* db, float* scratch, int T, int D, int accumulate,
                            void* stream) {
  return gf_layernorm_bwd_res(x, w, dy, mean, rstd, nullptr, dx, dw, db, scratch, T, D, accumulate, stream);
}
