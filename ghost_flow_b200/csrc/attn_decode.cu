// Single-query attention over a KV cache (the decode step of generation), grouped-query aware.
//
// The reference decodes by recomputing full attention on the CPU (ghostflow-nn/src/gpt.rs generate loop,
// ghostflow-nn/src/attention.rs:11-49). Here one CTA handles one KV head of a part of the keys (see DecWork); the G = Hq / Hkv
// <= 8 query heads that share the KV head are processed together, so each cache row is read once, and softmax is kept online.
// The pieces of a sequence are merged by a second kernel, which is on the machine before the first one ends. The cache read is
// the only traffic that matters, and what bounds the kernel is how much of it is in flight, and where: every warp has its own
// ring of DEC_STAGES blocks of 16 keys (K and V) filled by cp.async two blocks ahead, 128 KB on an SM, and neighbouring CTAs
// read the same keys of neighbouring heads, which are one piece of memory (a head's row is 256 bytes; with the CTAs of a
// sequence at different keys, 32 sequences of 4096 keys took 98 us instead of 86). A CTA that goes from one sequence to the
// next loses about 4 us of its own.
//
// The products run on mma.m16n8k16 with keys (S^T = K Q^T) and then head dimensions (O^T = V^T P^T) as the 16 rows and the
// query heads as the 8 columns, so no half of an instruction is padding, and the heads of a lane's scores are those of its
// output columns. K is read with ldmatrix, V with its transposing form, and P^T becomes the other operand with movmatrix.
// (tcgen05 tiles would need 128 query rows.) An operand has 8 bits and a probability 24, so P^T goes in as two bf16 numbers,
// the rounded value and what it left: the error of a result is then its own rounding to bf16 (0.00165 .. 0.00168 of the norm
// for both head sizes, as with P in fp32; rounded once, P makes it 0.0019 .. 0.0022). The second product costs 2 % where memory
// bounds the kernel (32 sequences of 1 .. 4096 keys, 32 / 8 heads of 128: 60.7 -> 61.5 us; 64 of 2048 keys, 64 / 8 heads: 90.0
// -> 92.1), 7 % where 160 to 240 CTAs leave SMs half empty; a third changes no digit. Device time with cold caches, us, a grid
// over sequences with slices of equal number / this: 32 sequences of 1 .. 4096 keys, 32 / 8 heads of 128 58.0 / 56.1 (shares),
// 8 of 1 .. 1501, 32 / 32 heads 23.6 / 19.5, 62 of 1 .. 300, 64 / 8 heads 28.5 / 15.4, 32 of 1 .. 4096, 12 / 12 heads of 64
// 44.9 / 41.1; one length: 32 of 4096, 32 / 8 heads 90.8 / 82.8 (6.5 TB/s), 8 of 1501, 32 / 32 heads 36.3 / 32.6, 8 of 4000, 40
// / 40 heads 112.2 / 103.9, 32 of 4096, 12 / 12 heads of 64 72.7 / 60.7 (6.6 TB/s), 64 of 300, 16 / 2 heads of 64 5.9 / 5.9, 4
// of 64, 64 / 8 heads of 64 3.1 / 3.2.
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

template <int D, bool SHARES>
struct DecCfg {
  static constexpr int ROW = D * 2;
  static constexpr int TILE = DEC_KEYS * ROW;          // K or V of a block
  static constexpr int WARP_BYTES = DEC_STAGES * 2 * TILE;
  static constexpr int RING = DEC_WARPS * WARP_BYTES;
  static constexpr int PITCH = D + 4;                  // a head's sums, maximum and total; the pitch spreads a lane's heads over the banks
  static constexpr int SMEM = RING + (SHARES ? 2 * DEC_MAX_G * PITCH * 4 : 0);
  static constexpr int CTAS = D > 64 ? 2 : 4;          // on an SM
  static_assert(DEC_WARPS * DEC_MAX_G * PITCH * 4 <= RING, "results fit in the ring");
  // 16-byte chunk c of row r lies at chunk c ^ (r % 8): ldmatrix meets every bank once, and rows fill whole lines
  __device__ __forceinline__ static int chunk(int row, int col) { return (col ^ (row & 7)) << 4; }
};

// How the keys are dealt out. A unit is 64 keys of one KV head (16 for each warp); an empty sequence has one. Neighbouring CTAs
// have the same keys of neighbouring KV heads, whose rows lie side by side in memory.
//   splits > 0   every sequence is cut into `splits` parts that differ by one unit at most. No merge with one part.
//   splits == 0  the sequences, one behind the other, are cut into `parts` parts that differ by one unit at most, whatever
//                the lengths are: a part may begin and end inside a sequence.
// A CTA has one KV head of one part. A piece that is not a whole sequence leaves its sums in a slot: the CTA's own (splits >
// 0), else the CTA's slot 0 where the sequence began in an earlier part and slot 1 where it began here and goes on in the next.
// A second kernel adds them up.
struct DecWork {
  const int* lens;
  int len_all, s_max, B, Hkv, parts, splits;
  __device__ __forceinline__ int len(int b) const { return lens ? max(0, min(lens[b], s_max)) : len_all; }
  __device__ __forceinline__ static int units(int len) { return max(1, (len + 63) >> 6); }
  // part of n equal ones (none empty: n <= total) that holds unit u
  __device__ __forceinline__ static int part_of(long long u, int n, int total) { return (int)(((u + 1) * n - 1) / total); }
};

// Whole warp: units before sequence b, and those of all sequences in `total`.
__device__ __forceinline__ int dec_units_before(const DecWork& w, int b, int& total) {
  if (!w.lens) {
    const int n = DecWork::units(w.len_all);
    total = n * w.B;
    return n * b;
  }
  const int lane = threadIdx.x & 31;
  int before = 0, all = 0;
  for (int i = lane; i < w.B; i += 32) {
    const int n = DecWork::units(w.len(i));
    all += n;
    if (i < b) before += n;
  }
  total = __reduce_add_sync(0xffffffffu, all);
  return __reduce_add_sync(0xffffffffu, before);
}

// A place in the order of the units of one KV head.
struct DecAt {
  int b, blk, len, n;
  __device__ __forceinline__ void next(const DecWork& w) {
    if (++blk < n) return;
    blk = 0;
    if (++b < w.B) {
      len = w.len(b);
      n = DecWork::units(len);
    }
  }
};

// Whole warp: the place of unit u < total.
__device__ __forceinline__ DecAt dec_find(const DecWork& w, int u) {
  DecAt at;
  if (!w.lens) {
    at.len = w.len_all;
    at.n = DecWork::units(at.len);
    at.b = u / at.n;
    at.blk = u - at.b * at.n;
    return at;
  }
  const int lane = threadIdx.x & 31;
  for (int base = 0, before = 0;; base += 32) {
    const int n = base + lane < w.B ? DecWork::units(w.len(base + lane)) : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, before + incl > u);
    if (hit || base + 32 >= w.B) {
      const int l = hit ? __ffs(hit) - 1 : 31;
      at.b = base + l;
      at.n = __shfl_sync(0xffffffffu, n, l);
      at.blk = u - before - (__shfl_sync(0xffffffffu, incl, l) - at.n);
      at.len = w.len(at.b);
      return at;
    }
    before += __shfl_sync(0xffffffffu, incl, 31);
  }
}

struct DecParams {
  DecWork work;
  const __nv_bfloat16* q;       // [B, Hq * D], pitch ldq; with append: packed rows [Hq + 2 Hkv heads of D]
  long long ldq;
  __nv_bfloat16 *kc, *vc;       // [B, s_max, Hkv * D]
  int Hq, G;                    // G = Hq / Hkv
  float scale_log2;
  float* part;                  // [slots][G heads][D sums, maximum, total]
  __nv_bfloat16* out;
  long long ldo;
  // append (gf_llama_decode): the new token's k and v are row len - 1; q and k are rotated here with these rows of the tables
  const float *cos_row, *sin_row;
  int interleaved;
};

// Rotates packed pairs: lo holds dims d, d + 1 and hi their partners (half-split), or each word is a pair (interleaved); the
// arithmetic and its rounding are the ones of rope_qkv_kernel.
__device__ __forceinline__ void rope_words(uint32_t& lo, uint32_t& hi, const float* c, const float* s, int d, int half,
                                           int interleaved) {
  const float2 a = unpack_bf16x2(lo), b = unpack_bf16x2(hi);
  if (interleaved) {
    const int i = d >> 1, j = (d + half) >> 1;
    lo = pack_bf16x2(a.x * c[i] - a.y * s[i], a.y * c[i] + a.x * s[i]);
    hi = pack_bf16x2(b.x * c[j] - b.y * s[j], b.y * c[j] + b.x * s[j]);
  } else {
    lo = pack_bf16x2(a.x * c[d] - b.x * s[d], a.y * c[d + 1] - b.y * s[d + 1]);
    hi = pack_bf16x2(b.x * c[d] + a.x * s[d], b.y * c[d + 1] + a.y * s[d + 1]);
  }
}

enum DecKind : int {
  DEC_SLICES = 0,    // splits > 0
  DEC_APPEND = 1,    // the same, with the new token's row
  DEC_SHARES = 2,    // splits == 0
};

// Kinds of one piece to a CTA are compiled without what goes from one sequence to the next. With it, calls that the memory does
// not bound took 5 to 25 % longer: us with / without it, 4 sequences of 64 keys, 64 / 8 heads of 64 3.8 / 3.1, 32 of 800, 32 /
// 8 heads of 64 13.7 / 11.4, 32 of 200, 32 / 32 heads of 128 32.7 / 26.5. (Padded rows instead of the exchange of chunks are 10
// % slower where memory bounds it: 32 of 4096 keys, 32 / 8 heads of 128 93 / 82: cp.async then fills lines in two parts.)
template <int D, int KIND>
__global__ void __launch_bounds__(DEC_WARPS * 32, DecCfg<D, KIND == DEC_SHARES>::CTAS)
attn_decode_kernel(const __grid_constant__ DecParams p) {
  constexpr bool SHARES = KIND == DEC_SHARES, APPEND = KIND == DEC_APPEND;
  using Cfg = DecCfg<D, SHARES>;
  extern __shared__ __align__(128) uint8_t ring[];
  const DecWork& w = p.work;
  const int G = p.G;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = lane >> 2, c = lane & 3;
  if (threadIdx.x == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int hk = blockIdx.x % w.Hkv, part = blockIdx.x / w.Hkv;
  DecAt at;
  int left_units;                  // of this CTA's part
  if constexpr (SHARES) {
    int total;
    dec_units_before(w, 0, total);
    const int parts = min(w.parts, total);                       // none is empty
    const int u0 = (int)((long long)part * total / parts);
    left_units = part < parts ? (int)((long long)(part + 1) * total / parts) - u0 : 0;
    if (left_units > 0) at = dec_find(w, u0);
  } else {
    at.b = part;
    if (w.splits > 1) at.b = part / w.splits;
    at.len = w.len(at.b);
    at.n = left_units = DecWork::units(at.len);
    at.blk = 0;
    if (w.splits > 1) {
      const unsigned sp = part - at.b * w.splits, splits = w.splits;             // sp n / splits in 32 bits: splits < 2^16
      const unsigned each = (unsigned)at.n / splits, rest = (unsigned)at.n - each * splits;
      at.blk = (int)(sp * each + sp * rest / splits);
      left_units = (int)((sp + 1) * each + (sp + 1) * rest / splits) - at.blk;
    }
  }
  if (left_units <= 0) return;
  const long long row_stride = (long long)w.Hkv * D, batch_stride = (long long)w.s_max * row_stride;
  const bool wide = ((reinterpret_cast<uintptr_t>(p.kc) | reinterpret_cast<uintptr_t>(p.vc)) & 15) == 0;   // rows are multiples of it
  const uint32_t my = smem_u32(ring) + warp * Cfg::WARP_BYTES;
  DecAt ahead = at;
  int ahead_units = left_units;
  long long head = at.b * batch_stride + (long long)hk * D;      // of the sequence ahead
  // keys of this warp's next unit into stage `st`; one commit group per unit, empty ones behind the part
  auto load = [&](int st) {
    const int k0 = ahead.blk * 64 + warp * DEC_KEYS;
    if (ahead_units > 0 && k0 < ahead.len) {
      const uint32_t dst = my + st * (2 * Cfg::TILE);
      const int lim = ahead.len - (APPEND ? 1 : 0);              // rows to read: the new token's comes from registers
#pragma unroll
      for (int n = 0; n < DEC_KEYS * D / 8 / 32; ++n) {
        const int id = lane + n * 32, row = id / (D / 8), col = id % (D / 8);
        const int key = k0 + row;
        const long long off = head + (long long)max(0, min(key, lim - 1)) * row_stride + col * 8;
        const uint32_t to = dst + row * Cfg::ROW + Cfg::chunk(row, col);
        if (wide) {
          const uint32_t bytes = key < lim ? 16u : 0u;
          cp_async_16(to, p.kc + off, bytes);
          cp_async_16(to + Cfg::TILE, p.vc + off, bytes);
        } else {                   // caches that start off a 16-byte boundary
          __nv_bfloat16* sk = reinterpret_cast<__nv_bfloat16*>(ring + (to - smem_u32(ring)));
#pragma unroll 1
          for (int e = 0; e < 8; ++e) {
            sk[e] = key < lim ? p.kc[off + e] : __float2bfloat16(0.f);
            sk[Cfg::TILE / 2 + e] = key < lim ? p.vc[off + e] : __float2bfloat16(0.f);
          }
        }
      }
    }
    --ahead_units;
    if constexpr (SHARES) {
      if (ahead_units > 0) {
        ahead.next(w);
        head = ahead.b * batch_stride + (long long)hk * D;
      }
    } else {
      ++ahead.blk;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < DEC_STAGES - 1; ++i) load(i);
  if (APPEND) asm volatile("griddepcontrol.wait;" ::: "memory");

  uint32_t qb[D / 16][2];          // Q^T as the 8-column operand: head r, dims 16 t + 2c, + 1 and + 8, + 9
  float o[D / 16][4];              // O^T: dims 16 j + r (+ 8), heads 2c, 2c + 1
  float m[2], l[2];
  uint4 k_new, v_new;              // append: chunk `lane` of the new token's rows, in the warp whose keys it belongs to
  // ---- start of a piece
  auto begin = [&] {
    const unsigned short* qp = reinterpret_cast<const unsigned short*>(
        p.q + at.b * p.ldq + (long long)(hk * G + min(r, G - 1)) * D + 2 * c);
#pragma unroll
    for (int t = 0; t < D / 16; ++t) {
      qb[t][0] = r < G ? qp[16 * t] | ((uint32_t)qp[16 * t + 1] << 16) : 0u;
      qb[t][1] = r < G ? qp[16 * t + 8] | ((uint32_t)qp[16 * t + 9] << 16) : 0u;
    }
    if (APPEND) {
      if (lane < D / 8) {
        const __nv_bfloat16* kn = p.q + at.b * p.ldq + (long long)(p.Hq + hk) * D;
        const int pc = (lane + D / 16) % (D / 8);                // the chunk half a head away
        k_new = *reinterpret_cast<const uint4*>(kn + lane * 8);
        v_new = *reinterpret_cast<const uint4*>(kn + (long long)w.Hkv * D + lane * 8);
        uint4 k_far = *reinterpret_cast<const uint4*>(kn + pc * 8);
        uint32_t *x = reinterpret_cast<uint32_t*>(&k_new), *y = reinterpret_cast<uint32_t*>(&k_far);
        const bool low = lane < D / 16;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          rope_words(low ? x[e] : y[e], low ? y[e] : x[e], p.cos_row, p.sin_row, (low ? lane : pc) * 8 + 2 * e, D / 2, p.interleaved);
      }
#pragma unroll
      for (int t = 0; t < D / 32; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          rope_words(qb[t][h], qb[t + D / 32][h], p.cos_row, p.sin_row, 16 * t + 2 * c + 8 * h, D / 2, p.interleaved);
    }
#pragma unroll
    for (int j = 0; j < D / 16; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    m[0] = m[1] = -INFINITY;
    l[0] = l[1] = 0.f;
  };
  // ---- the unit at `at`, in stage st
  auto unit = [&](int st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(DEC_STAGES - 1) : "memory");
    __syncwarp();
    const int left = at.len - (at.blk * 64 + warp * DEC_KEYS);    // valid keys of the block
    if (APPEND && left > 0 && left <= DEC_KEYS) {                 // the new token is the last valid key: into the ring and the caches
      if (lane < D / 8) {
        const int row = left - 1;
        uint8_t* to = ring + (my - smem_u32(ring)) + st * (2 * Cfg::TILE) + row * Cfg::ROW + Cfg::chunk(row, lane);
        *reinterpret_cast<uint4*>(to) = k_new;
        *reinterpret_cast<uint4*>(to + Cfg::TILE) = v_new;
        const long long off = at.b * batch_stride + (long long)(at.len - 1) * row_stride + (long long)hk * D + lane * 8;
        *reinterpret_cast<uint4*>(p.kc + off) = k_new;
        *reinterpret_cast<uint4*>(p.vc + off) = v_new;
      }
      __syncwarp();
    }
    if (left > 0) {
      const uint32_t tk = my + st * (2 * Cfg::TILE), tv = tk + Cfg::TILE;
      // S^T: keys r, r + 8 by heads 2c, 2c + 1
      float sc[4] = {0.f, 0.f, 0.f, 0.f}, sd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int t = 0; t < D / 16; ++t) {
        uint32_t a[4];
        ldmatrix_x4(a, tk + (lane & 15) * Cfg::ROW + Cfg::chunk(lane, 2 * t + (lane >> 4)));
        if (t & 1) mma_bf16_16816(sd, a[0], a[1], a[2], a[3], qb[t][0], qb[t][1]);
        else mma_bf16_16816(sc, a[0], a[1], a[2], a[3], qb[t][0], qb[t][1]);
      }
      float corr[2], pr[4];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float x0 = r < left ? (sc[e] + sd[e]) * p.scale_log2 : -INFINITY;
        const float x1 = r + 8 < left ? (sc[2 + e] + sd[2 + e]) * p.scale_log2 : -INFINITY;
        float mx = fmaxf(x0, x1);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
        const float mn = fmaxf(m[e], mx);
        const float ref = mn == -INFINITY ? 0.f : mn;      // every score so far -inf
        corr[e] = ex2_approx(m[e] - ref);
        m[e] = mn;
        pr[e] = ex2_approx(x0 - ref);
        pr[2 + e] = ex2_approx(x1 - ref);
        l[e] = l[e] * corr[e] + pr[e] + pr[2 + e];
      }
      uint32_t pt[DEC_P_TERMS][2];
#pragma unroll
      for (int n = 0; n < DEC_P_TERMS; ++n) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t x = pack_bf16x2(pr[2 * h], pr[2 * h + 1]);
          const float2 f = unpack_bf16x2(x);
          pr[2 * h] -= f.x;             // exact: what this term leaves
          pr[2 * h + 1] -= f.y;
          pt[n][h] = transpose_8x8(x);
        }
      }
      // O^T += V^T P^T
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        uint32_t a[4];
        ldmatrix_x4_trans(a, tv + ((lane & 7) + ((lane >> 4) << 3)) * Cfg::ROW + Cfg::chunk(lane, 2 * j + ((lane >> 3) & 1)));
        o[j][0] *= corr[0]; o[j][1] *= corr[1]; o[j][2] *= corr[0]; o[j][3] *= corr[1];
#pragma unroll
        for (int n = 0; n < DEC_P_TERMS; ++n) mma_bf16_16816(o[j], a[0], a[1], a[2], a[3], pt[n][0], pt[n][1]);
      }
    }
    __syncwarp();                  // the stage is filled again two units on
  };
  // ---- end of a piece: the warps' results meet, in the ring behind the CTA's last piece, else in two buffers of their own, in two
  // steps (2 and 3 give theirs to 0 and 1, then 1 to 0) while the ring fills with the next sequence. whole: the piece is a sequence
  auto finish = [&](const bool last, const bool whole, const long long slot_of) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      l[e] += __shfl_xor_sync(0xffffffffu, l[e], 4);
      l[e] += __shfl_xor_sync(0xffffffffu, l[e], 8);
      l[e] += __shfl_xor_sync(0xffffffffu, l[e], 16);
    }
    constexpr int BUF = DEC_MAX_G * Cfg::PITCH;
    float* buf = reinterpret_cast<float*>(ring + (last ? 0 : Cfg::RING));
    auto give = [&](float* to) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float* g = to + (2 * c + e) * Cfg::PITCH;
#pragma unroll
        for (int j = 0; j < D / 16; ++j) {
          g[16 * j + r] = o[j][e];
          g[16 * j + 8 + r] = o[j][2 + e];
        }
        if (r == 0) {
          g[D] = m[e];
          g[D + 1] = l[e];
        }
      }
    };
    if (last) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      give(buf + warp * BUF);
    } else {
      auto take = [&](const float* from) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float* g = from + (2 * c + e) * Cfg::PITCH;
          const float mo = g[D], mn = fmaxf(m[e], mo), ref = mn == -INFINITY ? 0.f : mn;
          const float ca = ex2_approx(m[e] - ref), cb = ex2_approx(mo - ref);
          m[e] = mn;
          l[e] = l[e] * ca + g[D + 1] * cb;
#pragma unroll
          for (int j = 0; j < D / 16; ++j) {
            o[j][e] = o[j][e] * ca + g[16 * j + r] * cb;
            o[j][2 + e] = o[j][2 + e] * ca + g[16 * j + 8 + r] * cb;
          }
        }
        __syncwarp();              // read by all lanes before the buffer is written again
      };
      if (warp >= 2) give(buf + (warp - 2) * BUF);
      __syncthreads();
      if (warp < 2) take(buf + warp * BUF);
      if (warp == 1) give(buf + BUF);
      __syncthreads();
      if (warp == 0) {
        take(buf + BUF);
        give(buf);
      }
    }
    __syncthreads();
    const int have = last ? DEC_WARPS : 1;
    __nv_bfloat16* to = p.out + at.b * p.ldo + (long long)hk * G * D;
    float* slot = p.part + slot_of * G * (D + 2);
    for (int i = threadIdx.x; i < G * D; i += DEC_WARPS * 32) {
      const int g = i / D, d = i % D;
      const float* x = buf + g * Cfg::PITCH;
      float mm = x[D], ll = x[D + 1], ov = x[d];
      if (have > 1) {
#pragma unroll
        for (int k = 1; k < DEC_WARPS; ++k) mm = fmaxf(mm, x[k * BUF + D]);
        const float ref = mm == -INFINITY ? 0.f : mm;
        float e = ex2_approx(x[D] - ref);
        ll *= e;
        ov *= e;
#pragma unroll
        for (int k = 1; k < DEC_WARPS; ++k) {
          e = ex2_approx(x[k * BUF + D] - ref);
          ll += x[k * BUF + D + 1] * e;
          ov += x[k * BUF + d] * e;
        }
      }
      if (whole) {
        to[i] = __float2bfloat16(ll > 0.f ? ov / ll : 0.f);
      } else {
        slot[g * (D + 2) + d] = ov;
        if (d == 0) {
          slot[g * (D + 2) + D] = mm;
          slot[g * (D + 2) + D + 1] = ll;
        }
      }
    }
  };

  int st = 0, st_load = DEC_STAGES - 1;
  if constexpr (!SHARES) {
    const bool whole = left_units == at.n;
    begin();
    for (; left_units > 0; --left_units, ++at.blk) {
      load(st_load);
      if (++st_load == DEC_STAGES) st_load = 0;
      unit(st);
      if (++st == DEC_STAGES) st = 0;
    }
    finish(true, whole, blockIdx.x);
  } else {
    bool begins = false;           // the piece in work starts with its head's first unit
    for (bool first = true; left_units > 0; first = false) {
      load(st_load);
      if (++st_load == DEC_STAGES) st_load = 0;
      if (first || at.blk == 0) {
        begins = at.blk == 0;
        begin();
      }
      unit(st);
      if (++st == DEC_STAGES) st = 0;
      const bool ends = at.blk == at.n - 1;
      if (ends || left_units == 1) {
        finish(left_units == 1, begins && ends, 2 * (long long)blockIdx.x + begins);
        __syncthreads();
      }
      if (--left_units > 0) at.next(w);
    }
  }
}

// One CTA of D threads for each query head: heads whose units all lay in one part are done, the others' pieces are added up,
// the loads of eight of them at a time.
template <int D>
__global__ void __launch_bounds__(D) attn_decode_merge_kernel(const __grid_constant__ DecParams p) {
  __shared__ float share[D];                       // exp2(maximum of piece k - maximum of all)
  const DecWork& w = p.work;
  const int G = p.G, b = blockIdx.x, h = blockIdx.y, hk = h / G, g = h - hk * G, d = threadIdx.x;
  const long long piece = (long long)G * (D + 2);
  const float *first, *rest;                       // the first piece's sums, and where piece k > 0 is: rest + k * step
  long long step;
  int pieces;
  const int n = DecWork::units(w.len(b));
  if (w.splits > 0) {
    pieces = min(n, w.splits);                     // with fewer units than parts some are empty
    step = w.Hkv * piece;
    first = rest = p.part + ((long long)b * w.splits * w.Hkv + hk) * piece + (long long)g * (D + 2);
  } else {
    int total;
    const int s0 = dec_units_before(w, b, total), parts = min(w.parts, total);
    const int c0 = DecWork::part_of(s0, parts, total), c1 = DecWork::part_of(s0 + n - 1, parts, total);
    pieces = c1 - c0 + 1;
    step = 2 * w.Hkv * piece;
    rest = p.part + ((long long)c0 * w.Hkv + hk) * 2 * piece + (long long)g * (D + 2);
    first = rest + piece;                          // slot 1 of its CTA
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (pieces == 1) return;
  auto at = [&](int k) -> const float* {
    if (w.splits > n) return rest + DecWork::part_of(k, w.splits, n) * step;
    return k ? rest + k * step : first;
  };
  if (pieces <= 8) {                               // one trip to memory
    float m[8], l[8], x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float* s = at(min(k, pieces - 1));
      m[k] = k < pieces ? s[D] : -INFINITY;
      l[k] = s[D + 1];
      x[k] = s[d];
    }
    float mm = m[0];
#pragma unroll
    for (int k = 1; k < 8; ++k) mm = fmaxf(mm, m[k]);
    const float ref = mm == -INFINITY ? 0.f : mm;
    float o = 0.f, t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float e = ex2_approx(m[k] - ref);
      o += x[k] * e;
      t += l[k] * e;
    }
    p.out[b * p.ldo + (long long)h * D + d] = __float2bfloat16(t > 0.f ? o / t : 0.f);
    return;
  }
  float mm = -INFINITY;
  for (int k = d & 31; k < pieces; k += 32) mm = fmaxf(mm, at(k)[D]);
#pragma unroll
  for (int o = 16; o; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
  const float ref = mm == -INFINITY ? 0.f : mm;
  float o = 0.f, l = 0.f;
  for (int k0 = 0; k0 < pieces; k0 += D) {
    __syncthreads();
    float e = 0.f;
    if (k0 + d < pieces) {
      const float* x = at(k0 + d);
      e = ex2_approx(x[D] - ref);
      l += e * x[D + 1];
    }
    share[d] = e;
    __syncthreads();
    const int m = min(D, pieces - k0);
    for (int k = 0; k < m; k += 8) {
      float x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = k + i < m ? at(k0 + k + i)[d] : 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) o += k + i < m ? x[i] * share[k + i] : 0.f;
    }
  }
  // the total of all pieces, the same in every thread
#pragma unroll
  for (int s = 16; s; s >>= 1) l += __shfl_xor_sync(0xffffffffu, l, s);
  __syncthreads();
  if ((d & 31) == 0) share[d >> 5] = l;
  __syncthreads();
  l = 0.f;
#pragma unroll
  for (int i = 0; i < D / 32; ++i) l += share[i];
  p.out[b * p.ldo + (long long)h * D + d] = __float2bfloat16(l > 0.f ? o / l : 0.f);
}

template <int D, int KIND>
static int launch_decode(const DecParams& p, int chained, cudaStream_t st) {
  static gf::DeviceOnce configured;
  constexpr int SMEM = DecCfg<D, KIND == DEC_SHARES>::SMEM;
  auto kern = attn_decode_kernel<D, KIND>;
  if (configured.todo()) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess)
      return GFH_CUDA;
    configured.mark();
  }
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.work.splits > 0 ? p.work.B * p.work.splits : p.work.parts) * p.work.Hkv));
  cfg.blockDim = dim3(DEC_WARPS * 32);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = chained ? 1 : 0;
  if (cudaLaunchKernelEx(&cfg, kern, p) != cudaSuccess) return GFH_CUDA;
  if (p.work.splits == 1) return GFH_OK;
  cfg.gridDim = dim3((unsigned)p.work.B, (unsigned)p.Hq);
  cfg.blockDim = dim3(D);
  cfg.dynamicSmemBytes = 0;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, attn_decode_merge_kernel<D>, p) != cudaSuccess) return GFH_CUDA;
  gf::note_extra_launches(1);
  return GFH_OK;
}

int attn_decode_append(const void* qkv, long long ldq, void* kcache, void* vcache, int s_max, int len, const float* cos_row,
                       const float* sin_row, int interleaved, void* out, long long ldo, int B, int Hq, int Hkv, int D, float scale,
                       int splits, float* scratch, int chained, cudaStream_t st) {
  if (B <= 0 || Hkv <= 0 || Hq % Hkv || Hq / Hkv > DEC_MAX_G || (D != 64 && D != 128) || splits < 1 || !scratch || len < 1 ||
      len > s_max || ldq % 8)
    return GFH_BAD_ARG;
  if (splits > 65535) splits = 65535;
  for (const void* x : {qkv, (const void*)kcache, (const void*)vcache})       // the new token's rows are read and written as vectors
    if (!x || (reinterpret_cast<uintptr_t>(x) & 15)) return GFH_BAD_ARG;
  DecParams p{{nullptr, len, s_max, B, Hkv, 0, splits}, (const __nv_bfloat16*)qkv, ldq, (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache,
              Hq, Hq / Hkv, scale * 1.4426950408889634f, scratch, (__nv_bfloat16*)out, ldo, cos_row, sin_row, interleaved};
  return D == 128 ? launch_decode<128, DEC_APPEND>(p, chained, st) : launch_decode<64, DEC_APPEND>(p, chained, st);
}

}  // namespace gf

using namespace gf;

// q [B, Hq * D] pitch ldq; caches [B, s_max, Hkv * D] contiguous; out [B, Hq * D] pitch ldo.
// `lens` (device int[B]) gives the valid length per sequence; nullptr: `len_all` for every sequence.
// splits > 0: parts of each sequence; scratch fp32 [B * Hq * splits * (D + 2)]. splits < 0: -splits parts of all sequences
// together; scratch fp32 [2 * -splits * Hq * (D + 2)].
GF_API int gf_attn_decode(const void* q, long long ldq, const void* kcache, const void* vcache, int s_max,
                          const int* lens, int len_all, void* out, long long ldo, int B, int Hq, int Hkv, int D,
                          float scale, int splits, float* scratch, void* stream) {
  gf::enter();
  if (B <= 0 || Hkv <= 0 || Hq % Hkv || Hq / Hkv > DEC_MAX_G || (D != 64 && D != 128) || splits == 0 || !scratch) return GFH_BAD_ARG;
  if (splits > 65535) splits = 65535;
  DecParams p{{lens, len_all, s_max, B, Hkv, splits < 0 ? -splits : 0, splits > 0 ? splits : 0}, (const __nv_bfloat16*)q, ldq,
              (__nv_bfloat16*)kcache, (__nv_bfloat16*)vcache,
              Hq, Hq / Hkv, scale * 1.4426950408889634f, scratch, (__nv_bfloat16*)out, ldo, nullptr, nullptr, 0};
  cudaStream_t st = (cudaStream_t)stream;
  if (splits < 0) return D == 128 ? launch_decode<128, DEC_SHARES>(p, 0, st) : launch_decode<64, DEC_SHARES>(p, 0, st);
  return D == 128 ? launch_decode<128, DEC_SLICES>(p, 0, st) : launch_decode<64, DEC_SLICES>(p, 0, st);
}
