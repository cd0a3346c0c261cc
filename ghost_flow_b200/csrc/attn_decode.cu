// Single-query attention over a KV cache (the decode step of generation), grouped-query aware.
//
// The reference decodes by recomputing full attention on the CPU (ghostflow-nn/src/gpt.rs generate loop,
// ghostflow-nn/src/attention.rs:11-49). Here one CTA handles one (sequence, KV head, slice of the cache); the G = Hq / Hkv <= 8
// query heads that share the KV head are processed together, so each cache row is read once, and softmax is kept online.
// Slices are merged by a second kernel (a single slice writes the result itself). The cache read is the only traffic
// that matters, and what bounds the kernel is how much of it is in flight: every warp has its own ring of DEC_STAGES blocks
// of 16 keys (K and V) filled by cp.async two blocks ahead, 128 KB on an SM. Loading K into registers, then V, one
// block at a time left the memory idle half of the time.
//
// The products run on mma.m16n8k16 with keys (S^T = K Q^T) and then head dimensions (O^T = V^T P^T) as the 16 rows and the
// query heads as the 8 columns, so no half of an instruction is padding, and the heads of a lane's scores are those of
// its output columns. K is read with ldmatrix, V with its transposing form, and P^T becomes the other operand with movmatrix.
// (tcgen05 tiles would need 128 query rows.)
// An operand has 8 bits and a probability 24, so P^T goes in as two bf16 numbers, the rounded value and what it left: the
// error of a result is then its own rounding to bf16 (0.00165 .. 0.00168 of the norm for both head sizes, as with P in fp32; rounded
// once, P makes it 0.0019 .. 0.0022). The second product costs 2 % where memory bounds the kernel (32 sequences of 1 .. 4096 keys,
// 32 / 8 heads of 128: 60.7 -> 61.5 us; 64 of 2048 keys, 64 / 8 heads: 90.0 -> 92.1), 7 % where 160 to 240 CTAs leave SMs half
// empty; a third changes no digit.
// Measured, before -> now: 32 sequences of 1 .. 4096 keys, 32 / 8 heads of 128 77 -> 58 us (4.4 TB/s); 8 sequences of
// 1501 keys, 32 / 32 heads of 128 58 -> 38 us; 64 of 2048 keys, 64 / 8 heads 156 -> 92 us (5.8 TB/s); 8 of 4000 keys, 40 / 40
// heads 133 -> 115 us (5.7 TB/s); 32 of 1 .. 4096 keys, 12 / 12 heads of 64 295 -> 44 us (those went one key at a time).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "gf_host.h"
#include "gf_ptx.cuh"

namespace gf {

constexpr int DEC_WARPS = 4;
constexpr int DEC_MAX_G = 8;
constexpr int DEC_KEYS = 16;     // keys of a block
constexpr int DEC_STAGES = 3;
constexpr int DEC_P_TERMS = 2;   // bf16 numbers that stand for a probability

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
// 16 bytes global -> shared; `bytes` = 0 writes zeros instead (the source is not read)
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int D>
struct DecCfg {
  static constexpr int ROW = D * 2 + 16;               // padded row: ldmatrix meets every bank once
  static constexpr int TILE = DEC_KEYS * ROW;          // K or V of a block
  static constexpr int WARP_BYTES = DEC_STAGES * 2 * TILE;
  static constexpr int SMEM = DEC_WARPS * WARP_BYTES;  // reused for the warps' results
  static_assert(SMEM >= DEC_WARPS * DEC_MAX_G * (D + 2) * 4, "results fit in the ring");
};

// q [B, Hq * D] (pitch ldq), k/v cache [B, s_max, Hkv * D]; part_o [B, Hq, splits, D] fp32, part_ml [B, Hq, splits, 2];
// out [B, Hq * D] (pitch ldo) when there is one slice.
template <int D>
__global__ void __launch_bounds__(DEC_WARPS * 32, 2)
attn_decode_kernel(const __nv_bfloat16* __restrict__ q, long long ldq, const __nv_bfloat16* __restrict__ kc,
                   const __nv_bfloat16* __restrict__ vc, long long batch_stride, long long row_stride,
                   const int* __restrict__ lens, int len_all, int Hq, int Hkv, float scale_log2,
                   float* __restrict__ part_o, float* __restrict__ part_ml, int splits, __nv_bfloat16* __restrict__ out,
                   long long ldo) {
  using Cfg = DecCfg<D>;
  extern __shared__ __align__(16) uint8_t ring[];
  const int b = blockIdx.x, hk = blockIdx.y, sp = blockIdx.z;
  const int G = Hq / Hkv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane >> 2, c = lane & 3;
  const int len = lens ? lens[b] : len_all;
  const int chunk = (len + splits - 1) / splits;
  const int s0 = sp * chunk, s1 = min(len, s0 + chunk);

  const __nv_bfloat16* kb = kc + (long long)b * batch_stride + (long long)hk * D;
  const __nv_bfloat16* vb = vc + (long long)b * batch_stride + (long long)hk * D;
  const bool wide = ((reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) == 0;   // rows are multiples of it
  const uint32_t my = smem_u32(ring) + warp * Cfg::WARP_BYTES;
  // block i of this warp: keys s0 + (4 i + warp) * 16 ..; one commit group per block, empty ones behind the slice
  auto load = [&](int i) {
    const int k0 = s0 + (i * DEC_WARPS + warp) * DEC_KEYS;
    if (k0 < s1) {
      const uint32_t dst = my + (i % DEC_STAGES) * (2 * Cfg::TILE);
#pragma unroll
      for (int n = 0; n < DEC_KEYS * D / 8 / 32; ++n) {
        const int id = lane + n * 32, row = id / (D / 8), col = id % (D / 8);
        const int key = k0 + row;
        const long long off = (long long)min(key, s1 - 1) * row_stride + col * 8;
        const uint32_t at = dst + row * Cfg::ROW + col * 16;
        if (wide) {
          const uint32_t bytes = key < s1 ? 16u : 0u;
          cp_async_16(at, kb + off, bytes);
          cp_async_16(at + Cfg::TILE, vb + off, bytes);
        } else {                   // caches that start off a 16-byte boundary
          __nv_bfloat16* sk = reinterpret_cast<__nv_bfloat16*>(ring + (at - smem_u32(ring)));
#pragma unroll 1
          for (int e = 0; e < 8; ++e) {
            sk[e] = key < s1 ? kb[off + e] : __float2bfloat16(0.f);
            sk[Cfg::TILE / 2 + e] = key < s1 ? vb[off + e] : __float2bfloat16(0.f);
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < DEC_STAGES - 1; ++i) load(i);

  uint32_t qb[D / 16][2];          // Q^T as the 8-column operand: head r, dims 16 t + 2c, + 1 and + 8, + 9
#pragma unroll
  for (int t = 0; t < D / 16; ++t) {
    const unsigned short* qp = reinterpret_cast<const unsigned short*>(
        q + (long long)b * ldq + (long long)(hk * G + min(r, G - 1)) * D + 16 * t + 2 * c);
    qb[t][0] = r < G ? qp[0] | ((uint32_t)qp[1] << 16) : 0u;
    qb[t][1] = r < G ? qp[8] | ((uint32_t)qp[9] << 16) : 0u;
  }
  float o[D / 16][4];              // O^T: dims 16 j + r (+ 8), heads 2c, 2c + 1
#pragma unroll
  for (int j = 0; j < D / 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

  for (int i = 0; s0 + (i * DEC_WARPS + warp) * DEC_KEYS < s1; ++i) {
    load(i + DEC_STAGES - 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(DEC_STAGES - 1) : "memory");
    __syncwarp();
    const uint32_t tk = my + (i % DEC_STAGES) * (2 * Cfg::TILE), tv = tk + Cfg::TILE;
    // ---- S^T: keys r, r + 8 by heads 2c, 2c + 1
    float sc[4] = {0.f, 0.f, 0.f, 0.f}, sd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int t = 0; t < D / 16; ++t) {
      uint32_t a[4];
      ldmatrix_x4(a, tk + (lane & 15) * Cfg::ROW + (16 * t + (lane >> 4) * 8) * 2);
      if (t & 1) mma_bf16_16816(sd, a[0], a[1], a[2], a[3], qb[t][0], qb[t][1]);
      else mma_bf16_16816(sc, a[0], a[1], a[2], a[3], qb[t][0], qb[t][1]);
    }
    const int left = s1 - (s0 + (i * DEC_WARPS + warp) * DEC_KEYS);    // valid keys of the block, at least one
    float corr[2], p[4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float x0 = r < left ? (sc[e] + sd[e]) * scale_log2 : -INFINITY;
      const float x1 = r + 8 < left ? (sc[2 + e] + sd[2 + e]) * scale_log2 : -INFINITY;
      float mx = fmaxf(x0, x1);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
      const float mn = fmaxf(m[e], mx);
      const float ref = mn == -INFINITY ? 0.f : mn;      // every score so far -inf
      corr[e] = ex2_approx(m[e] - ref);
      m[e] = mn;
      p[e] = ex2_approx(x0 - ref);
      p[2 + e] = ex2_approx(x1 - ref);
      l[e] = l[e] * corr[e] + p[e] + p[2 + e];
    }
    uint32_t pt[DEC_P_TERMS][2];
#pragma unroll
    for (int n = 0; n < DEC_P_TERMS; ++n) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t u = pack_bf16x2(p[2 * h], p[2 * h + 1]);
        const float2 f = unpack_bf16x2(u);
        p[2 * h] -= f.x;             // exact: what this term leaves
        p[2 * h + 1] -= f.y;
        pt[n][h] = transpose_8x8(u);
      }
    }
    // ---- O^T += V^T P^T
#pragma unroll
    for (int j = 0; j < D / 16; ++j) {
      uint32_t a[4];
      ldmatrix_x4_trans(a, tv + ((lane & 7) + ((lane >> 4) << 3)) * Cfg::ROW + (16 * j + ((lane >> 3) & 1) * 8) * 2);
      o[j][0] *= corr[0]; o[j][1] *= corr[1]; o[j][2] *= corr[0]; o[j][3] *= corr[1];
#pragma unroll
      for (int n = 0; n < DEC_P_TERMS; ++n) mma_bf16_16816(o[j], a[0], a[1], a[2], a[3], pt[n][0], pt[n][1]);
    }
    __syncwarp();                  // the stage is filled again two blocks on
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    l[e] += __shfl_xor_sync(0xffffffffu, l[e], 4);
    l[e] += __shfl_xor_sync(0xffffffffu, l[e], 8);
    l[e] += __shfl_xor_sync(0xffffffffu, l[e], 16);
  }
  // ---- the four warps' results meet in the ring's memory
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* sm_acc = reinterpret_cast<float*>(ring);                      // [warp][head][D]
  float* sm_ml = sm_acc + DEC_WARPS * DEC_MAX_G * D;                   // [warp][head][2]
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int g = warp * DEC_MAX_G + 2 * c + e;
#pragma unroll
    for (int j = 0; j < D / 16; ++j) {
      sm_acc[g * D + 16 * j + r] = o[j][e];
      sm_acc[g * D + 16 * j + 8 + r] = o[j][2 + e];
    }
    if (r == 0) {
      sm_ml[g * 2] = m[e];
      sm_ml[g * 2 + 1] = l[e];
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < G * D; idx += DEC_WARPS * 32) {
    const int g = idx / D, dd = idx % D;
    float mm = -INFINITY;
    for (int w = 0; w < DEC_WARPS; ++w) mm = fmaxf(mm, sm_ml[(w * DEC_MAX_G + g) * 2]);
    float ll = 0.f, ov = 0.f;
    for (int w = 0; w < DEC_WARPS; ++w) {
      const float mw = sm_ml[(w * DEC_MAX_G + g) * 2];
      const float cw = mw == -INFINITY ? 0.f : ex2_approx(mw - mm);
      ll += sm_ml[(w * DEC_MAX_G + g) * 2 + 1] * cw;
      ov += sm_acc[(w * DEC_MAX_G + g) * D + dd] * cw;
    }
    if (splits == 1) {
      out[(long long)b * ldo + (long long)(hk * G + g) * D + dd] = __float2bfloat16(ll > 0.f ? ov / ll : 0.f);
    } else {
      const long long base = ((long long)b * Hq + hk * G + g) * splits + sp;
      part_o[base * D + dd] = ov;
      if (dd == 0) { part_ml[base * 2] = mm; part_ml[base * 2 + 1] = ll; }
    }
  }
}

template <int D>
__global__ void attn_decode_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                         __nv_bfloat16* __restrict__ out, long long ldo, int Hq, int splits) {
  const int b = blockIdx.x, h = blockIdx.y, dd = threadIdx.x;
  const long long base = ((long long)b * Hq + h) * splits;
  float mm = -INFINITY;
  for (int s = 0; s < splits; ++s) mm = fmaxf(mm, part_ml[(base + s) * 2]);
  float ll = 0.f, o = 0.f;
  for (int s = 0; s < splits; ++s) {
    const float ms = part_ml[(base + s) * 2];
    const float c = ms == -INFINITY ? 0.f : ex2_approx(ms - mm);
    ll += part_ml[(base + s) * 2 + 1] * c;
    o += part_o[(base + s) * D + dd] * c;
  }
  out[(long long)b * ldo + (long long)h * D + dd] = __float2bfloat16(ll > 0.f ? o / ll : 0.f);
}

template <int D>
static int launch_decode(const void* q, long long ldq, const void* kc, const void* vc, long long batch, long long row,
                         const int* lens, int len_all, void* out, long long ldo, int B, int Hq, int Hkv, float sl2, int splits,
                         float* scratch, cudaStream_t st) {
  static gf::DeviceOnce configured;
  if (configured.todo()) {
    if (cudaFuncSetAttribute(attn_decode_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, DecCfg<D>::SMEM) !=
        cudaSuccess)
      return GFH_CUDA;
    configured.mark();
  }
  float* part_o = scratch;
  float* part_ml = scratch + (long long)B * Hq * splits * D;
  attn_decode_kernel<D><<<dim3(B, Hkv, splits), DEC_WARPS * 32, DecCfg<D>::SMEM, st>>>(
      (const __nv_bfloat16*)q, ldq, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc, batch, row, lens, len_all, Hq, Hkv,
      sl2, part_o, part_ml, splits, (__nv_bfloat16*)out, ldo);
  if (splits > 1) {
    attn_decode_merge_kernel<D><<<dim3(B, Hq), D, 0, st>>>(part_o, part_ml, (__nv_bfloat16*)out, ldo, Hq, splits);
    gf::note_extra_launches(1);
  }
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

}  // namespace gf

using namespace gf;

// q [B, Hq * D] pitch ldq; caches [B, s_max, Hkv * D] contiguous; out [B, Hq * D] pitch ldo.
// `lens` (device int[B]) gives the valid length per sequence; nullptr: `len_all` for every sequence.
// scratch: fp32 [B * Hq * splits * (D + 2)].
GF_API int gf_attn_decode(const void* q, long long ldq, const void* kcache, const void* vcache, int s_max,
                          const int* lens, int len_all, void* out, long long ldo, int B, int Hq, int Hkv, int D,
                          float scale, int splits, float* scratch, void* stream) {
  gf::enter();
  if (B <= 0 || Hq % Hkv || Hq / Hkv > DEC_MAX_G || (D != 64 && D != 128) || splits < 1 || !scratch) return GFH_BAD_ARG;
  const long long row = (long long)Hkv * D, batch = (long long)s_max * row;
  const float sl2 = scale * 1.4426950408889634f;
  auto launch = D == 128 ? launch_decode<128> : launch_decode<64>;
  return launch(q, ldq, kcache, vcache, batch, row, lens, len_all, out, ldo, B, Hq, Hkv, sl2, splits, scratch,
                (cudaStream_t)stream);
}
