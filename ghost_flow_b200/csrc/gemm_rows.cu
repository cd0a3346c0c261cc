// bf16 GEMM of a few rows (one token of each sequence of a batch): C[M, N] = act(alpha * f(X)[M, K] W[N, K]^T + bias +
// residual), M <= 64.
//
// The weight is read once and is all that counts, so it is the 128-row operand: tcgen05.mma with 128 output features as the
// rows and 16, 32 or 64 tokens as the columns. TMA fills a ring of 128 x 64 weight blocks, about 200 KB on an SM for its two or
// three CTAs, and needs no registers for what is in flight. K is split over the CTAs of a cluster; they add their sums through
// distributed shared memory in the order of their ranks, so there is no workspace to clear, no atomic and no second kernel.
//
// The tokens' side of a block comes by TMA too, or (at most 16 rows) four warps compute it, so that the operation in front of
// the product needs no launch and no trip through memory: an RMS norm (the operand is x * w rounded to bf16, and the row's
// factor 1 / rms scales the sums; the squares are added up from the same loads) or SwiGLU. The norm costs 0.2 us. SwiGLU, an
// exponential and a division for each element in every CTA that reads it, costs more than the 2 us of its own kernel: [1,
// 28672] x [8192, 28672]^T 73 -> 106 us, [8, 11008] x [4096, 11008]^T 19.4 -> 26.1, [1, 688] x [256, 688]^T 5.6 -> 8.6; the
// decoder layer uses the kernel. With more rows each CTA would compute more than it has time for beside its weights: fused, 64
// rows of a LLaMA-7B layer took 286 us, with a norm kernel in front 214.
//
// In a chain of launches the weight blocks are on their way before the kernel in front has finished (griddepcontrol): they are
// nobody's output there. X, the residual and C are touched behind griddepcontrol.wait only.
//
// What bounds it: memory, behind a fixed cost of about 5 us (launch, TMEM, first block, cluster barriers). The rings hold up to
// 28 MB in flight. Up to 16 tokens three smaller CTAs share an SM: more of them mean shorter parts of K and a better fit to the
// machine (a layer of 8 sequences, hidden 4096 / 5120: two CTAs of six stages 121 / 134 us, three of four 116 / 112; half as
// many CTAs 138 / 182). Device time in us with cold weights, the kernels that took these products before -> this one: [16,
// 4096] x [12288, 4096]^T 27.0 -> 20.8 (4.8 TB/s), x [22016, 4096]^T 40.9 -> 33.2 (5.4 TB/s), [16, 11008] x [4096, 11008]^T
// 24.0 -> 19.7; back to back from the host [32, 4096] x [22016, 4096]^T 54.2 -> 41.9, [64, 4096] x [4096, 4096]^T 21.9 -> 14.7,
// [64, 14336] x [8192, 14336]^T 55.6 -> 45.8.
#include <atomic>

#include "gemm_rows.cuh"
#include "gf_host.h"
#include "gf_ptx.cuh"

namespace gf {

constexpr int RW_BM = 128;                  // features of a tile
constexpr int RW_BK = 64;
constexpr int RW_THREADS = 192;             // TMA warp, MMA warp, four warps for the tokens and the epilogue
constexpr int RW_W_BYTES = RW_BM * RW_BK * 2;

template <int NT>
struct RwCfg {
  static constexpr int X_BYTES = NT * RW_BK * 2;
  static constexpr int STAGE_BYTES = RW_W_BYTES + X_BYTES;
  static constexpr int STAGES = NT == 32 ? 5 : 4;
  static constexpr int CTAS = NT == 16 ? 3 : 2;                       // on an SM
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 512;
  static constexpr int TMEM_COLS = NT < 32 ? 32 : NT;
  static_assert(NT * RW_BM * 4 <= STAGES * STAGE_BYTES, "partial sums fit in the ring");
};

struct RowsParams {
  const __nv_bfloat16* X;
  long long ldx;
  void* C;
  long long ldc;
  int out_fp32, M, N, K;
  const __nv_bfloat16* norm_w;
  float eps;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  float alpha;
  int relu;
  int quads;       // C and residual rows on boundaries of four values, N a multiple of four
  int* status;
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ float4 ld_peer_f32x4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ float ld_peer_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ float silu_mul(float g, float u) { return g * (1.f / (1.f + __expf(-g))) * u; }

template <int NT, int INPUT>
__global__ void __launch_bounds__(RW_THREADS, RwCfg<NT>::CTAS)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                 const __grid_constant__ RowsParams p) {
  using Cfg = RwCfg<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + Cfg::STAGES;
  uint64_t* acc_full = empty + Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  float* row_sum = reinterpret_cast<float*>(acc_full + 2);       // [NT] squares of this CTA's part of K, then the row factors

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t rank, ranks;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(ranks));
  const int n0 = (int)(blockIdx.x / ranks) * RW_BM;
  const int blocks = (p.K + RW_BK - 1) / RW_BK;
  const int kb0 = (int)(rank * (unsigned)blocks / ranks), kb1 = (int)((rank + 1) * (unsigned)blocks / ranks);

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full[s], INPUT == ROWS_PLAIN ? 1 : 1 + 4);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (threadIdx.x == 0) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (warp == 0) {
    if (lane == 0) {
      // weight blocks for the whole ring first, then (plain input) the tokens' blocks beside them once they may be read
      constexpr uint32_t BYTES = INPUT == ROWS_PLAIN ? Cfg::STAGE_BYTES : RW_W_BYTES;
      const int first = min(Cfg::STAGES, kb1 - kb0);
      for (int i = 0; i < first; ++i) {
        mbar_expect_tx(&full[i], BYTES);
        tma_load_2d(smem + i * Cfg::STAGE_BYTES, &tmW, &full[i], (kb0 + i) * RW_BK, n0);
      }
      if (INPUT == ROWS_PLAIN) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        for (int i = 0; i < first; ++i)
          tma_load_2d(smem + i * Cfg::STAGE_BYTES + RW_W_BYTES, &tmX, &full[i], (kb0 + i) * RW_BK, 0);
      }
      int st = 0;
      uint32_t ph = 0;
      for (int kb = kb0 + Cfg::STAGES; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[st], ph)) {
          if (p.status) atomicCAS(p.status, 0, GF_ERR_WAIT_EMPTY);
          break;
        }
        mbar_expect_tx(&full[st], BYTES);
        tma_load_2d(smem + st * Cfg::STAGE_BYTES, &tmW, &full[st], kb * RW_BK, n0);
        if (INPUT == ROWS_PLAIN) tma_load_2d(smem + st * Cfg::STAGE_BYTES + RW_W_BYTES, &tmX, &full[st], kb * RW_BK, 0);
        if (++st == Cfg::STAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(RW_BM, NT, 0, 0);
    int st = 0;
    uint32_t ph = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp_tight(&full[st], ph)) {
        if (p.status && leader) atomicCAS(p.status, 0, GF_ERR_WAIT_FULL);
        break;
      }
      tc_fence_after();
      const uint32_t base = smem_u32(smem + st * Cfg::STAGE_BYTES);
      const uint64_t wd = umma_desc_sw128(base, 16, 1024), xd = umma_desc_sw128(base + RW_W_BYTES, 16, 1024);
#pragma unroll
      for (int kk = 0; kk < RW_BK / 16; ++kk)
        umma_bf16_ss_u(leader, tmem, wd + kk * 2, xd + kk * 2, idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
      umma_commit_u(leader, &empty[st]);
      if (++st == Cfg::STAGES) { st = 0; ph ^= 1; }
    }
    umma_commit_u(leader, acc_full);
  } else {
    // ---------------------------------------------------------------- tokens of a block: eight threads to a 128-byte row
    const int tid = threadIdx.x - 64;
    const int vec = tid & 7, tok = tid >> 3;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    bool ok = true;
    if constexpr (INPUT != ROWS_PLAIN) {
      static_assert(NT == 16, "a vector of a block for each of 128 threads");
      constexpr int B = 2;                 // blocks whose loads are issued together
      float sq = 0.f;
      uint4 x[2][B], y[2][B];              // y: up projection, or the norm's weight
      auto load = [&](int kb, uint4 (&xr)[B], uint4 (&yr)[B]) {
#pragma unroll
        for (int i = 0; i < B; ++i) {
          const int k = (kb + i) * RW_BK + vec * 8;
          const bool in = kb + i < kb1 && k < p.K;             // K is a multiple of eight
          const __nv_bfloat16* src = p.X + (long long)tok * p.ldx + k;
          xr[i] = in && tok < p.M ? *reinterpret_cast<const uint4*>(src) : make_uint4(0, 0, 0, 0);
          if (INPUT == ROWS_SWIGLU) yr[i] = in && tok < p.M ? *reinterpret_cast<const uint4*>(src + p.K) : make_uint4(0, 0, 0, 0);
          if (INPUT == ROWS_RMSNORM) yr[i] = in ? *reinterpret_cast<const uint4*>(p.norm_w + k) : make_uint4(0, 0, 0, 0);
        }
      };
      int st = 0;
      uint32_t ph = 1;
      auto store = [&](int kb, const uint4 (&xr)[B], const uint4 (&yr)[B]) {
#pragma unroll
        for (int i = 0; i < B; ++i) {
          if (kb + i >= kb1 || !ok) break;
          if (!mbar_wait_warp_tight(&empty[st], ph)) {
            if (p.status && lane == 0) atomicCAS(p.status, 0, GF_ERR_WAIT_EMPTY);
            ok = false;
            break;
          }
          uint4 o = xr[i];
          uint32_t* po = reinterpret_cast<uint32_t*>(&o);
          const uint32_t* pw = reinterpret_cast<const uint32_t*>(&yr[i]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 a = unpack_bf16x2(po[e]), w = unpack_bf16x2(pw[e]);
            if (INPUT == ROWS_RMSNORM) {
              sq += a.x * a.x + a.y * a.y;
              po[e] = pack_bf16x2(a.x * w.x, a.y * w.y);
            } else {
              po[e] = pack_bf16x2(silu_mul(a.x, w.x), silu_mul(a.y, w.y));
            }
          }
          *reinterpret_cast<uint4*>(smem + st * Cfg::STAGE_BYTES + RW_W_BYTES + sw128_offset(tok, vec)) = o;
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[st]);
          if (++st == Cfg::STAGES) { st = 0; ph ^= 1; }
        }
      };
      load(kb0, x[0], y[0]);
      for (int kb = kb0; kb < kb1 && ok; kb += 2 * B) {
        load(kb + B, x[1], y[1]);
        store(kb, x[0], y[0]);
        load(kb + 2 * B, x[0], y[0]);
        store(kb + B, x[1], y[1]);
      }
      if (INPUT == ROWS_RMSNORM) {
        sq += __shfl_xor_sync(0xffffffffu, sq, 1);
        sq += __shfl_xor_sync(0xffffffffu, sq, 2);
        sq += __shfl_xor_sync(0xffffffffu, sq, 4);
        if (vec == 0) row_sum[tok] = sq;
      }
    }
    // ---------------------------------------------------------------- sums of this CTA: [token][feature] over the ring
    if (ok && !mbar_wait_warp_tight(acc_full, 0)) {
      if (p.status && lane == 0) atomicCAS(p.status, 0, GF_ERR_WAIT_TMEM_FULL);
      ok = false;
    }
    if (ok) {
      tc_fence_after();
      float* part = reinterpret_cast<float*>(smem);
      const int f = (warp & 3) * 32 + lane;
#pragma unroll
      for (int c = 0; c < NT / 16; ++c) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c * 16, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) part[(c * 16 + i) * RW_BM + f] = __uint_as_float(r[i]);
      }
    }
  }
  if (p.status && *reinterpret_cast<volatile int*>(p.status) != 0) error_drain_pause();
  __syncwarp();
  tc_fence_before();
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  if (warp >= 2) {
    const uint32_t part = smem_u32(smem), sums = smem_u32(row_sum);
    uint32_t peer[8];
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q)
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer[q]) : "r"(part), "r"(q < ranks ? q : 0u));
    // The rows of the tile are dealt to the warps of all ranks in turn; a lane has four features of a row. The loads of ROWS
    // rows are issued before the first is used: one row at a time, 64 rows cost 30 us.
    constexpr int ROWS = 4;
    const int f = lane * 4, n = n0 + f, step = 4 * (int)ranks;
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if (p.bias)
      for (int e = 0; e < 4; ++e)
        if (n + e < p.N) bias[e] = __bfloat162float(p.bias[n + e]);
    for (int m0 = (int)rank * 4 + warp - 2; m0 < p.M; m0 += ROWS * step) {
      float4 v[ROWS];
      float sq[ROWS];
      uint2 res[ROWS];
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int m = m0 + i * step;
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        sq[i] = 0.f;
        res[i] = make_uint2(0u, 0u);
        if (m >= p.M) continue;
        if (p.residual && p.quads && n < p.N) res[i] = *reinterpret_cast<const uint2*>(p.residual + (long long)m * p.ldr + n);
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q) {
          if (q < ranks) {
            const float4 a = ld_peer_f32x4(peer[q] + (uint32_t)(m * RW_BM + f) * 4);
            v[i].x += a.x; v[i].y += a.y; v[i].z += a.z; v[i].w += a.w;
            if (INPUT == ROWS_RMSNORM) sq[i] += ld_peer_f32(peer[q] + (sums - part) + (uint32_t)m * 4);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int m = m0 + i * step;
        if (m >= p.M || n >= p.N) continue;
        const float k = INPUT == ROWS_RMSNORM ? p.alpha * rsqrtf(sq[i] / (float)p.K + p.eps) : p.alpha;
        float y[4] = {v[i].x * k + bias[0], v[i].y * k + bias[1], v[i].z * k + bias[2], v[i].w * k + bias[3]};
        if (p.quads) {
          if (p.residual) {
            const float2 a = unpack_bf16x2(res[i].x), b = unpack_bf16x2(res[i].y);
            y[0] += a.x; y[1] += a.y; y[2] += b.x; y[3] += b.y;
          }
          if (p.relu) {
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = fmaxf(y[e], 0.f);
          }
          if (p.out_fp32)
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + (long long)m * p.ldc + n) =
                make_float4(y[0], y[1], y[2], y[3]);
          else
            *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)m * p.ldc + n) =
                make_uint2(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]));
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (n + e >= p.N) break;
            float t = y[e];
            if (p.residual) t += __bfloat162float(p.residual[(long long)m * p.ldr + n + e]);
            if (p.relu) t = fmaxf(t, 0.f);
            if (p.out_fp32) reinterpret_cast<float*>(p.C)[(long long)m * p.ldc + n + e] = t;
            else reinterpret_cast<__nv_bfloat16*>(p.C)[(long long)m * p.ldc + n + e] = __float2bfloat16(t);
          }
        }
      }
    }
  }
  // no CTA leaves while another one may still read its sums
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::TMEM_COLS);
  }
}

bool gemm_rows_takes(const void* X, long long ldx, const void* W, long long ldw, int M, int N, int K) {
  return M > 0 && M <= ROWS_MAX_M && N > 0 && K > 0 && K % 8 == 0 && ldx % 8 == 0 && ldw % 8 == 0 &&
         ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
}

static void rows_attributes(cudaLaunchConfig_t& cfg, cudaLaunchAttribute (&at)[2], int grid, int smem, int slices, int chained) {
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(RW_THREADS);
  cfg.dynamicSmemBytes = smem;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)slices; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained ? 2 : 1;
}

// Never launched: the CTAs of this one share an SM as those of the kernel do (shared memory is what counts), and are counted
// so. For a kernel with tensor memory the runtime counts one CTA to an SM.
template <int NT>
__global__ void __launch_bounds__(RW_THREADS, RwCfg<NT>::CTAS) rows_occupancy_kernel(int* p) {
  extern __shared__ int part[];
  if (p) *p = part[threadIdx.x];
}

// Clusters of `slices` CTAs that the current device holds at once: fewer than SMs x CTAs / slices, since a cluster lies within a
// GPC. Asked once for each size and device.
template <int NT>
static int rows_clusters(int slices) {
  using Cfg = RwCfg<NT>;
  static std::atomic<int> known[64][4];
  std::atomic<int>& k = known[gf::DeviceOnce::device()][slices >= 8 ? 3 : slices >> 1];
  int n = k.load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    rows_attributes(cfg, at, slices * sm_count() * Cfg::CTAS, Cfg::SMEM_BYTES, slices, 0);
    auto kern = rows_occupancy_kernel<NT>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      return sm_count() * Cfg::CTAS / slices;
    }
    k.store(n, std::memory_order_relaxed);
  }
  return n;
}

// CTAs of a cluster, each with a part of K of at least four blocks: as many as leave all clusters on the machine at once, and a
// power of two (clusters of 3, 6 or 7 leave SMs of a GPC out: 6144 features on 48 clusters of 6 took 22.4 us, on 48 of 4 14.7).
// Up to 16 tokens 48 clusters of 8 fit, 104 of 4, 222 of 2; with more tokens 33, 71 and 148. One more is a second wave: [8,
// 4096] x [N, 4096]^T, N = 6272 17.1 us on 49 of 8, 13.7 on 49 of 4; 13824 27.6 on 108 of 4, 22.7 on 108 of 2; 24 tokens, 4352
// 16.0 on 34 of 8, 12.0 on 34 of 4; 9216 23.9 on 72 of 4, 17.7 on 72 of 2. Tiles that do not fit at once even whole: the last
// ones stream all of K from a few CTAs, so a long K is cut in two where they are few (up to 16 tokens, where the second half
// overlaps with more, always). us whole / in two: [8, 8192] x [57344, 8192]^T (448 tiles) 162.1 / 146.7, x [73728, 8192]^T
// 180.7 / 176.8, x [128256, 8192]^T 303.2 / 301.1; K 4096: 83.4 / 77.1, 95.6 / 92.1, 158.0 / 152.6; K 2048: 45.4 / 45.4, 51.5 /
// 53.6; 24 tokens, K 8192: [38016] 119.0 / 107.8, [43008] 124.9 / 116.1, [57344] 144.4 / 152.2; 64 tokens [57344] 155.7 /
// 172.5.
template <int NT>
static int rows_slices(int N, int K) {
  const int tiles = (N + RW_BM - 1) / RW_BM, blocks = (K + RW_BK - 1) / RW_BK, whole = rows_clusters<NT>(1);
  if (tiles > whole) return blocks >= 64 && (NT == 16 || (tiles - 1) % whole < whole / 4) ? 2 : 1;
  int s = 8;
  while (s > 1 && (4 * s > blocks || tiles > rows_clusters<NT>(s))) s >>= 1;
  return s;
}

template <int NT, int INPUT>
static int launch_rows(const CUtensorMap& tm, const CUtensorMap& tx, const RowsParams& p, int chained, cudaStream_t stream) {
  using Cfg = RwCfg<NT>;
  auto kern = gemm_rows_kernel<NT, INPUT>;
  static gf::DeviceOnce configured;
  if (configured.todo()) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess)
      return GFH_CUDA;
    configured.mark();
  }
  const int slices = rows_slices<NT>(p.N, p.K);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  rows_attributes(cfg, at, (p.N + RW_BM - 1) / RW_BM * slices, Cfg::SMEM_BYTES, slices, chained);
  cfg.stream = stream;
  return cudaLaunchKernelEx(&cfg, kern, tm, tx, p) == cudaSuccess ? GFH_OK : GFH_CUDA;
}

template <int INPUT>
static int launch_rows_nt(const CUtensorMap& tm, const CUtensorMap& tx, const RowsParams& p, int chained, cudaStream_t stream) {
  if (p.M <= 16) return launch_rows<16, INPUT>(tm, tx, p, chained, stream);
  if constexpr (INPUT != ROWS_PLAIN) return GFH_BAD_ARG;
  else if (p.M <= 32) return launch_rows<32, INPUT>(tm, tx, p, chained, stream);
  else return launch_rows<64, INPUT>(tm, tx, p, chained, stream);
}

// What the kernel reads as 16-byte vectors beside X and W, and the kinds that there are.
static bool gemm_rows_input_ok(const RowsGemm& g) {
  if (g.input == ROWS_PLAIN) return true;
  if (g.M > ROWS_MAX_M_FUSED) return false;
  return g.input == ROWS_SWIGLU || (g.input == ROWS_RMSNORM && g.norm_w && (reinterpret_cast<uintptr_t>(g.norm_w) & 15) == 0);
}

int gemm_rows_run(const RowsGemm& g, int chained, cudaStream_t stream) {
  if (!gemm_rows_takes(g.X, g.ldx, g.W, g.ldw, g.M, g.N, g.K) || !gemm_rows_input_ok(g)) return GFH_BAD_ARG;
  CUtensorMap tm;
  const int rc = make_tmap_2d(&tm, g.W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, g.N, g.K, g.ldw * 2, RW_BM, RW_BK);
  if (rc) return rc;
  const int size = g.out_fp32 ? 16 : 8;
  const int quads = g.N % 4 == 0 && g.ldc % 4 == 0 && reinterpret_cast<uintptr_t>(g.C) % size == 0 &&
                    (!g.residual || (g.ldr % 4 == 0 && reinterpret_cast<uintptr_t>(g.residual) % 8 == 0));
  RowsParams p{(const __nv_bfloat16*)g.X, g.ldx, g.C, g.ldc, g.out_fp32, g.M, g.N, g.K, (const __nv_bfloat16*)g.norm_w, g.eps,
               (const __nv_bfloat16*)g.bias, (const __nv_bfloat16*)g.residual, g.ldr, g.alpha, g.relu, quads, g.status};
  if (g.input == ROWS_RMSNORM) return launch_rows_nt<ROWS_RMSNORM>(tm, tm, p, chained, stream);
  if (g.input == ROWS_SWIGLU) return launch_rows_nt<ROWS_SWIGLU>(tm, tm, p, chained, stream);
  CUtensorMap tx;
  const uint32_t rows = g.M <= 16 ? 16 : g.M <= 32 ? 32 : 64;
  const int rx = make_tmap_2d(&tx, g.X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, g.M, g.K, g.ldx * 2, rows, RW_BK);
  if (rx) return rx;
  return launch_rows_nt<ROWS_PLAIN>(tm, tx, p, chained, stream);
}

}  // namespace gf

// C[M, N] = act(alpha * f(X) W^T + bias + residual) of a few rows; see RowsGemm and RowsInput.
GF_API int gf_gemm_rows(const void* X, long long ldx, const void* W, long long ldw, void* C, long long ldc, int out_fp32, int M, int N,
                        int K, int input, const void* norm_w, float eps, const void* bias, const void* residual, long long ldr,
                        float alpha, int relu, int* status, void* stream) {
  gf::enter();
  gf::RowsGemm g{X, ldx, W, ldw, C, ldc, out_fp32, M, N, K, (gf::RowsInput)input, norm_w, eps, bias, residual, ldr, alpha, relu, status};
  return gf::gemm_rows_run(g, 0, (cudaStream_t)stream);
}

// On the current device: the CTAs of a cluster that such a product takes (slices = 0), or the clusters of `slices`
// CTAs that are on the machine at once.
GF_API int gf_gemm_rows_clusters(int M, int N, int K, int slices) {
  using namespace gf;
  if (M < 1 || M > ROWS_MAX_M || N < 1 || K < 1 || slices < 0 || slices > 8 || (slices & (slices - 1))) return GFH_BAD_ARG;
  bind();
  if (slices)
    return M <= 16 ? rows_clusters<16>(slices) : M <= 32 ? rows_clusters<32>(slices) : rows_clusters<64>(slices);
  return M <= 16 ? rows_slices<16>(N, K) : M <= 32 ? rows_slices<32>(N, K) : rows_slices<64>(N, K);
}
