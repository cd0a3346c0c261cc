// FlashAttention backward, third generation: one CTA owns a 128-row KV tile of one KV head and walks the 128-row query
// tiles that can see it. Per step, on tcgen05 with TMEM accumulators:
//     S^T = K Q^T, dP^T = V dO^T          128 x 128 x HD, operands from shared memory
//     dV += P^T dO                        128 x HD x 128, P^T as operand from tensor memory
//     dQ^T = K^T dS^T, dK += dS^T Q       HD x 128 x 128 and 128 x HD x 128, dS^T from shared memory
//
// 128-row steps need 40 instructions with N = 128 (64 cycles of the tensor pipe each, in every operand form) where 64-row
// steps needed 56, some with N = 64 that shared memory feeds at two thirds of the rate, and twice the waits, whose cold
// code between the unrolled loops of the other warps is what an MMA warp spends its time on. With dK and dV resident
// there is no tensor memory left to double-buffer S^T and dP^T at this size, so the order of the products keeps the
// pipe fed instead:
//     dP(i)  dV(i)  S(i + 1) | dQ(i)  dK(i)
// P(i) is computed under dQ(i - 1), dK(i - 1) and dP(i), dS(i) under dV(i) and S(i + 1), and dQ(i) is drained under dK(i).
// Regions of tensor memory are reused under these rules (MMAs of the one issuing thread execute in issue order):
//     columns   0..127  S^T, then P^T (bf16, packed into the first half of each compute group's own columns); S(i + 1) is
//                       issued after dV(i), which read P(i), and p_full(i), after which no warp reads S(i)
//     columns 128..255  dP^T, then dQ^T of the step, issued after ds_full(i), when no warp reads dP(i) any more; dP(i + 1)
//                       waits until the drain warps have dQ(i) in registers
//     columns 256..     dV, dK
// The one dS^T tile in shared memory is free again when dP(i + 1) is announced, since its commit also covers dK(i).
//
// dQ leaves through the bulk-copy engine: the drain warps transpose some query rows at a time through one of four staging
// tiles, and each is one fp32 add-reduction (cp.reduce.async.bulk) of a contiguous block of the accumulator
// [B, Hq, S, HD]. The softmax scale is taken out of the loop (dK gets it in the epilogue, dQ in the conversion kernel); the
// row statistics arrive as -lse * log2(e) and -delta, so that an element costs half a two-wide FMA, an exponential, half
// a two-wide addition and multiplication and two halves of a conversion.
//
// What bounds it: with HD = 128 the fp32 additions of dQ in L2 (a step's 64 KB take the drain warps 3500 of its 3600 to
// 3900 cycles, whatever the order of the products and the number of staging tiles; the tensor pipe needs 2560); with
// HD = 64 the chain dS -> dQ -> drain -> dP -> dS of about 2900 cycles a step.
//
// Measured, all launches of the backward pass, before -> now: [1, 4096, 32 heads of 128] causal 579 -> 398 us,
// [8, 1024, 12 heads of 64] causal 190 -> 126 us, [2, 4096, 16 heads of 128] full 974 -> 664 us, [16, 512, 16 / 4 heads of
// 128] causal 216 -> 144 us.
//
// The reference only names a backward kernel (ghostflow-cuda/src/kernels/mod.rs:82) and has no backward for its
// CPU flash attention (ghostflow-nn/src/flash_attention.rs).
#include "gf_host.h"
#include "gf_ptx.cuh"

namespace gf {

constexpr int B3_TILE = 128;      // kv rows per CTA, query rows per step
constexpr int B3_THREADS = 512;   // warpgroup 0: TMA warp, MMA warp, two idle; 1 and 2: compute; 3: dQ drain
// 128 x (104 + 2 x 136 + 136) = 65536 registers, the block's own at launch (512 x 128). No part spills with these; with 56
// for the first warpgroup the MMA warp reloaded descriptors from local memory between its instructions.
constexpr int B3_REGS_CTRL = 104;
constexpr int B3_REGS_COMPUTE = 136;
constexpr int B3_REGS_DRAIN = 136;

struct FaBwd3Params {
  int B, S, Hq, Hkv;
  int causal;
  float scale;
  const float* nlse2;   // [B, Hq, S]  -lse * log2(e)
  const float* ndelta;  // [B, Hq, S]  -sum_d O dO
  float* dq_acc;        // fp32 [B, Hq, S, HD], zero before launch; receives dQ / scale
  __nv_bfloat16* dK;
  long long lddk;
  __nv_bfloat16* dV;
  long long lddv;
  int* status;
  int head_group;       // KV heads (of all sequences) whose CTAs are dispatched together
};

template <int HD>
struct FaBwd3Cfg {
  static constexpr int CH = HD / 64;
  static constexpr int TILE_BYTES = B3_TILE * HD * 2;             // K, V, Q or dO tile
  static constexpr int DS_BYTES = B3_TILE * B3_TILE * 2;          // dS^T: two chunks of [128 kv rows][64 query columns]
  static constexpr int QST = HD == 64 ? 3 : 2;                    // Q and statistics stages
  static constexpr int STAGE_ROWS = HD == 64 ? 32 : 16;           // query rows of a staging tile
  static constexpr int STAGES_DQ = 4;
  static constexpr int DQ_BYTES = STAGE_ROWS * HD * 4;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + TILE_BYTES;                // directly behind K: see K_LBO
  static constexpr int OFF_Q = OFF_V + TILE_BYTES;                // QST stages
  static constexpr int OFF_DO = OFF_Q + QST * TILE_BYTES;
  static constexpr int OFF_DS = OFF_DO + TILE_BYTES;
  static constexpr int OFF_DQS = OFF_DS + DS_BYTES;               // STAGES_DQ staging tiles
  static constexpr int OFF_STAT = OFF_DQS + STAGES_DQ * DQ_BYTES; // QST stages x (nlse2[128], ndelta[128])
  static constexpr int OFF_BAR = OFF_STAT + QST * 2 * B3_TILE * 4;
  static constexpr int SMEM_BYTES = OFF_BAR + 256;
  static constexpr int TM_S = 0, TM_DP = 128, TM_DV = 256, TM_DK = 384;
  static constexpr int TMEM_COLS = 512;
};

template <int HD>
__global__ void __launch_bounds__(B3_THREADS, 1)
fa_bwd3_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
               const FaBwd3Params p) {
  using Cfg = FaBwd3Cfg<HD>;
  extern __shared__ __align__(1024) uint8_t smem[];   // the kernel has no other shared memory: the base is aligned
  if (smem_u32(smem) & 1023u) {
    if (p.status && threadIdx.x == 0) atomicCAS(p.status, 0, GF_ERR_BAD_ARG);
    return;
  }
  uint8_t* sK = smem + Cfg::OFF_K;
  uint8_t* sV = smem + Cfg::OFF_V;
  uint8_t* sQ = smem + Cfg::OFF_Q;
  uint8_t* sDO = smem + Cfg::OFF_DO;
  uint8_t* sDS = smem + Cfg::OFF_DS;
  float* sStat = reinterpret_cast<float*>(smem + Cfg::OFF_STAT);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* kv_full = bars + 0;
  uint64_t* acc_full = bars + 1;
  uint64_t* do_full = bars + 2;
  uint64_t* do_empty = bars + 3;
  uint64_t* s_full = bars + 4;
  uint64_t* p_full = bars + 5;      // P^T in tensor memory
  uint64_t* dp_full = bars + 6;
  uint64_t* ds_full = bars + 7;     // dS^T in shared memory
  uint64_t* dq_full = bars + 8;
  uint64_t* dq_empty = bars + 9;    // dQ^T in the drain warps' registers
  uint64_t* q_full = bars + 10;     // [QST]  Q tile and row statistics
  uint64_t* q_empty = q_full + Cfg::QST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(q_empty + Cfg::QST);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Linear block order: the KV heads of all sequences in groups of head_group; inside a group the heaviest KV tile of
  // every head first (under a causal mask tile 0 is seen by every query tile, the last one by one), so the CTAs in flight
  // share the Q / dO tiles of one group in L2 and the short CTAs fill the tail.
  int j, hk, b;
  {
    const int H = gridDim.x, NT = gridDim.y;
    const int lin = blockIdx.x + H * blockIdx.y;
    const int gs = p.head_group;
    const int g = lin / (gs * NT);
    const int rem = lin - g * gs * NT;
    const int gs_g = min(gs, H - g * gs);
    j = rem / gs_g;
    hk = g * gs + rem % gs_g;
    b = hk / p.Hkv;
    hk -= b * p.Hkv;
  }
  const int G = p.Hq / p.Hkv;
  const int i_start = p.causal ? j : 0;
  const int per_head = p.S / B3_TILE - i_start;
  const int n_iter = G * per_head;
  const int row_base = b * p.S;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    mbar_init(acc_full, 1);
    for (int i = 0; i < Cfg::QST; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(p_full, 8);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, 8);
    mbar_init(dq_full, 1);
    mbar_init(dq_empty, 4);
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(B3_REGS_CTRL));
    if (warp == 0) {
      // -------------------------------------------------------------- TMA producer
      if (lane == 0) {
        mbar_expect_tx(kv_full, 2 * Cfg::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < Cfg::CH; ++c) {
          tma_load_2d(sK + c * (B3_TILE * 128), &tmK, kv_full, hk * HD + c * 64, row_base + j * B3_TILE);
          tma_load_2d(sV + c * (B3_TILE * 128), &tmV, kv_full, hk * HD + c * 64, row_base + j * B3_TILE);
        }
        int h = hk * G, i = i_start - 1;
        int st = -1;
        uint32_t ph = 0;
        for (int it = 0; it < n_iter; ++it) {
          if (++st == Cfg::QST) { st = 0; ph ^= 1; }
          if (++i == i_start + per_head) { i = i_start; ++h; }
          if (!mbar_wait(&q_empty[st], ph ^ 1)) {
            if (p.status) atomicCAS(p.status, 0, GF_ERR_WAIT_EMPTY);
            break;
          }
          mbar_expect_tx(&q_full[st], Cfg::TILE_BYTES + 2 * B3_TILE * 4);
#pragma unroll
          for (int c = 0; c < Cfg::CH; ++c)
            tma_load_2d(sQ + st * Cfg::TILE_BYTES + c * (B3_TILE * 128), &tmQ, &q_full[st], h * HD + c * 64,
                        row_base + i * B3_TILE);
          const long long soff = ((long long)b * p.Hq + h) * p.S + (long long)i * B3_TILE;
          bulk_load_1d(sStat + st * 2 * B3_TILE, p.nlse2 + soff, B3_TILE * 4, &q_full[st]);
          bulk_load_1d(sStat + st * 2 * B3_TILE + B3_TILE, p.ndelta + soff, B3_TILE * 4, &q_full[st]);
          if (!mbar_wait(do_empty, (it & 1) ^ 1)) {
            if (p.status) atomicCAS(p.status, 0, GF_ERR_WAIT_EMPTY);
            break;
          }
          mbar_expect_tx(do_full, Cfg::TILE_BYTES);
#pragma unroll
          for (int c = 0; c < Cfg::CH; ++c)
            tma_load_2d(sDO + c * (B3_TILE * 128), &tmDO, do_full, h * HD + c * 64, row_base + i * B3_TILE);
        }
      }
    } else if (warp == 1) {
      // -------------------------------------------------------------- MMA issuer
      // The whole warp runs this code in uniform control flow; one elected lane issues (see gf_ptx.cuh).
      const bool leader = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, B3_TILE, 0, 0);   // S^T, dP^T
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, HD, 0, 1);      // dV, dK
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, B3_TILE, 1, 1);  // dQ^T
      constexpr uint64_t TILE_D = Cfg::TILE_BYTES >> 4;                   // descriptor addresses count 16-byte units
      // K^T as an MN-major operand: 64 head dimensions to a chunk. HD = 64: rows 64..127 of dQ^T read the V tile behind K
      // and are never drained
      constexpr uint32_t K_LBO = B3_TILE * 128;
      const uint64_t k_k = umma_desc_sw128(smem_u32(sK), 16, 1024), v_k = umma_desc_sw128(smem_u32(sV), 16, 1024);
      const uint64_t k_mn = umma_desc_sw128(smem_u32(sK), K_LBO, 1024);
      const uint64_t q_k = umma_desc_sw128(smem_u32(sQ), 16, 1024), do_k = umma_desc_sw128(smem_u32(sDO), 16, 1024);
      const uint64_t q_mn = umma_desc_sw128(smem_u32(sQ), B3_TILE * 128, 1024);
      const uint64_t do_mn = umma_desc_sw128(smem_u32(sDO), B3_TILE * 128, 1024);
      const uint64_t ds_k = umma_desc_sw128(smem_u32(sDS), 16, 1024);
      const uint64_t ds_mn = umma_desc_sw128(smem_u32(sDS), B3_TILE * 128, 1024);
      // offset of a Q stage, by selection: as a product of the loop-carried stage number it came out wrong for HD = 128
      // (nvcc 12.9, found by the fp64 test: every step after a CTA's first read the wrong columns)
      auto q_off = [](int st) -> uint64_t { return st == 0 ? 0 : st == 1 ? TILE_D : 2 * TILE_D; };
      int err = GF_OK;
      // S^T of the step whose Q is in stage st
      auto issue_s = [&](int st) {
        tc_fence_after();
        const uint64_t qd = q_k + q_off(st);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * (B3_TILE * 128) + (kk & 3) * 32) >> 4;
          umma_bf16_ss_u(leader, tmem_base + Cfg::TM_S, k_k + off, qd + off, idesc_s, kk > 0 ? 1u : 0u);
        }
        umma_commit_u(leader, s_full);
      };
      if (!mbar_wait_warp_tight(kv_full, 0)) err = GF_ERR_WAIT_FULL;
      if (err == GF_OK && n_iter > 0) {
        if (!mbar_wait_warp_tight(&q_full[0], 0)) err = GF_ERR_WAIT_FULL;
        else issue_s(0);
      }
      int st = 0;                          // stage of Q(it), and of Q(it + 1) with the parity of its use
#pragma unroll 1
      for (int it = 0, nx = 0, nph = 0; it < n_iter && err == GF_OK; ++it, st = nx) {
        if (++nx == Cfg::QST) { nx = 0; nph ^= 1; }
        if (!mbar_wait_warp_tight(do_full, it & 1)) { err = GF_ERR_WAIT_FULL; break; }
        if (!mbar_wait_warp_tight(dq_empty, (it & 1) ^ 1)) { err = GF_ERR_WAIT_TMEM_EMPTY; break; }
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) {
          const uint64_t off = ((kk >> 2) * (B3_TILE * 128) + (kk & 3) * 32) >> 4;
          umma_bf16_ss_u(leader, tmem_base + Cfg::TM_DP, v_k + off, do_k + off, idesc_s, kk > 0 ? 1u : 0u);
        }
        umma_commit_u(leader, dp_full);
        if (!mbar_wait_warp_tight(p_full, it & 1)) { err = GF_ERR_WAIT_SOFTMAX; break; }
        tc_fence_after();
        // dV += P^T dO: k step kk covers query columns 16 kk .., packed at column 64 (kk / 4) + 8 (kk % 4)
#pragma unroll
        for (int kk = 0; kk < B3_TILE / 16; ++kk)
          umma_bf16_ts_u(leader, tmem_base + Cfg::TM_DV, tmem_base + Cfg::TM_S + (kk >> 2) * 64 + (kk & 3) * 8,
                         do_mn + ((kk * 2048) >> 4), idesc_acc, (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit_u(leader, do_empty);
        if (it + 1 < n_iter) {
          if (!mbar_wait_warp_tight(&q_full[nx], nph)) { err = GF_ERR_WAIT_FULL; break; }
          issue_s(nx);
        }
        if (!mbar_wait_warp_tight(ds_full, it & 1)) { err = GF_ERR_WAIT_SOFTMAX; break; }
        tc_fence_after();
        // dQ^T first: it is drained while dK runs
#pragma unroll
        for (int kk = 0; kk < B3_TILE / 16; ++kk)
          umma_bf16_ss_u(leader, tmem_base + Cfg::TM_DP, k_mn + ((kk * 2048) >> 4), ds_mn + ((kk * 2048) >> 4), idesc_dq,
                         kk > 0 ? 1u : 0u);
        umma_commit_u(leader, dq_full);
        // dK += dS^T Q
        const uint64_t qd = q_mn + q_off(st);
#pragma unroll
        for (int kk = 0; kk < B3_TILE / 16; ++kk)
          umma_bf16_ss_u(leader, tmem_base + Cfg::TM_DK, ds_k + (((kk >> 2) * (B3_TILE * 128) + (kk & 3) * 32) >> 4),
                         qd + ((kk * 2048) >> 4), idesc_acc, (it > 0 || kk > 0) ? 1u : 0u);
        umma_commit_u(leader, &q_empty[st]);
      }
      if (err == GF_OK) umma_commit_u(leader, acc_full);
      else if (p.status && leader) atomicCAS(p.status, 0, err);
    }
  } else if (warp >= 12) {
    // ---------------------------------------------------------------- dQ drain warps (12..15)
    // Warp w owns TMEM lanes 32 * (w % 4) .. +31 = head-dim rows of dQ^T, 128 query columns per thread. STAGE_ROWS query
    // rows at a time go to a staging tile as [rows][HD] (a warp stores 32 consecutive floats, no bank conflicts).
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(B3_REGS_DRAIN));
    const int lane_grp = warp & 3;
    const int d = lane_grp * 32 + lane;
    const uint32_t tlane = (uint32_t)(lane_grp * 32) << 16;
    const bool issuer = (warp == 12 && lane == 0);
    int h = hk * G, i = i_start - 1;
    for (int it = 0; it < n_iter; ++it) {
      if (++i == i_start + per_head) { i = i_start; ++h; }
      // The four warps meet at named barriers below, so they must agree on giving up: the outcome of the
      // bounded wait is AND-reduced over the warpgroup (itself a barrier that every warp reaches).
      uint32_t all_ok;
      {
        const uint32_t mine = mbar_wait(dq_full, it & 1) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.u32 p, %1, 0;\n\t"
            "bar.red.and.pred q, 1, 128, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}\n"
            : "=r"(all_ok)
            : "r"(mine)
            : "memory");
      }
      if (!all_ok) {
        if (p.status) atomicCAS(p.status, 0, GF_ERR_WAIT_TMEM_FULL);
        break;
      }
      tc_fence_after();
      uint32_t rq[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(tmem_base + Cfg::TM_DP + c * 32 + tlane, rq[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_empty);
      float* tile = p.dq_acc + (((long long)b * p.Hq + h) * p.S + (long long)i * B3_TILE) * HD;
#pragma unroll
      for (int c = 0; c < B3_TILE / Cfg::STAGE_ROWS; ++c) {
        float* stage = reinterpret_cast<float*>(smem + Cfg::OFF_DQS + (c % Cfg::STAGES_DQ) * Cfg::DQ_BYTES);
        // the reduction that used this staging tile last has read it
        if (issuer) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(Cfg::STAGES_DQ - 1) : "memory");
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (d < HD) {
#pragma unroll
          for (int e = 0; e < Cfg::STAGE_ROWS; ++e) {
            const int q = c * Cfg::STAGE_ROWS + e;
            stage[e * HD + d] = __uint_as_float(rq[q >> 5][q & 31]);
          }
        }
        fence_proxy_async_smem();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (issuer) {
          asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(
                           tile + c * Cfg::STAGE_ROWS * HD),
                       "r"(smem_u32(stage)), "r"((uint32_t)Cfg::DQ_BYTES)
                       : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    // the reductions must have left shared memory (and be performed) before the CTA exits
    if (issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    // ---------------------------------------------------------------- compute warps (4..11)
    // Warps 4..7 own query columns 0..63 of S^T / dP^T, warps 8..11 columns 64..127; within a group, warp w owns
    // TMEM lanes 32 * (w % 4) .. +31, one kv row per thread.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(B3_REGS_COMPUTE));
    const int hf = (warp >> 2) - 1;
    const int lane_grp = warp & 3;
    const int r = lane_grp * 32 + lane;
    const uint32_t tlane = (uint32_t)(lane_grp * 32) << 16;
    const uint32_t ts = tmem_base + Cfg::TM_S + hf * 64 + tlane, tdp = tmem_base + Cfg::TM_DP + hf * 64 + tlane;
    const float sl2 = p.scale * 1.4426950408889634f;
    const uint64_t sl2x = pk2f(sl2, sl2);
    uint8_t* sDSh = sDS + hf * (B3_TILE * 128);
    bool ok = true;

    int i = i_start - 1, st = -1;
    uint32_t ph = 0;
#pragma unroll 1
    for (int it = 0; it < n_iter && ok; ++it) {
      if (++st == Cfg::QST) { st = 0; ph ^= 1; }
      if (++i == i_start + per_head) i = i_start;
      // the statistics arrive on q_full, the scores on s_full
      if (!mbar_wait_warp_tight(&q_full[st], ph) || !mbar_wait_warp_tight(s_full, it & 1)) {
        if (p.status) atomicCAS(p.status, 0, GF_ERR_WAIT_TMEM_FULL);
        ok = false;
        break;
      }
      tc_fence_after();
      const ulonglong2* nl = reinterpret_cast<const ulonglong2*>(sStat + st * 2 * B3_TILE + hf * 64);
      const ulonglong2* nd = reinterpret_cast<const ulonglong2*>(sStat + st * 2 * B3_TILE + B3_TILE + hf * 64);
      const bool diag = p.causal && i == j;
      uint64_t pr[32];   // P^T of this thread's row, two query columns to an entry, in fp32
      {
        uint32_t sv[2][32];
        tmem_ld32(ts, sv[0]);
        tmem_ld32(ts + 32, sv[1]);
        tmem_ld_wait();
#pragma unroll
        for (int e4 = 0; e4 < 16; ++e4) {
          const ulonglong2 n4 = nl[e4];
          const uint32_t* s4 = &sv[e4 >> 3][(e4 & 7) * 4];
          const uint64_t x0 = f2_fma(pk2(s4[0], s4[1]), sl2x, n4.x), x1 = f2_fma(pk2(s4[2], s4[3]), sl2x, n4.y);
          pr[e4 * 2] = pk2f(ex2_approx(lo2(x0)), ex2_approx(hi2(x0)));
          pr[e4 * 2 + 1] = pk2f(ex2_approx(lo2(x1)), ex2_approx(hi2(x1)));
        }
      }
      if (diag) {   // query column before the kv row: not visible
        const int lim = r - hf * 64;
#pragma unroll
        for (int e = 0; e < 32; ++e)
          pr[e] = pk2f(2 * e < lim ? 0.f : lo2(pr[e]), 2 * e + 1 < lim ? 0.f : hi2(pr[e]));
      }
      {
        uint32_t pp[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) pp[e] = pack_bf16x2(lo2(pr[e]), hi2(pr[e]));
        tmem_st32(ts, pp);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      if (!mbar_wait_warp_tight(dp_full, it & 1)) {
        if (p.status) atomicCAS(p.status, 0, GF_ERR_WAIT_TMEM_FULL);
        ok = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t dv[32], dd[16];
        tmem_ld32(tdp + c * 32, dv);
        tmem_ld_wait();
#pragma unroll
        for (int e4 = 0; e4 < 8; ++e4) {
          const ulonglong2 n4 = nd[c * 8 + e4];
          const uint64_t d0 = f2_mul(pr[c * 16 + e4 * 2], f2_add(pk2(dv[e4 * 4], dv[e4 * 4 + 1]), n4.x));
          const uint64_t d1 = f2_mul(pr[c * 16 + e4 * 2 + 1], f2_add(pk2(dv[e4 * 4 + 2], dv[e4 * 4 + 3]), n4.y));
          dd[e4 * 2] = pack_bf16x2(lo2(d0), hi2(d0));
          dd[e4 * 2 + 1] = pack_bf16x2(lo2(d1), hi2(d1));
        }
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4)
          *reinterpret_cast<uint4*>(sDSh + sw128_offset((uint32_t)r, (uint32_t)(c * 4 + c4))) =
              make_uint4(dd[c4 * 4], dd[c4 * 4 + 1], dd[c4 * 4 + 2], dd[c4 * 4 + 3]);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    if (ok) {
      if (!mbar_wait_warp_tight(acc_full, 0)) {
        if (p.status) atomicCAS(p.status, 0, GF_ERR_WAIT_TMEM_FULL);
      } else {
        tc_fence_after();
        const int kv_idx = j * B3_TILE + r;
        __nv_bfloat16* dkr = p.dK + (long long)(row_base + kv_idx) * p.lddk + hk * HD;
        __nv_bfloat16* dvr = p.dV + (long long)(row_base + kv_idx) * p.lddv + hk * HD;
        // each group writes half of the head dimension; dK gets the softmax scale here
#pragma unroll
        for (int cc = 0; cc < HD / 64; ++cc) {
          const int c = hf * (HD / 64) + cc;
          uint32_t rk[32], rv[32];
          tmem_ld32(tmem_base + Cfg::TM_DK + c * 32 + tlane, rk);
          tmem_ld32(tmem_base + Cfg::TM_DV + c * 32 + tlane, rv);
          tmem_ld_wait();
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 uk, uv;
            uint32_t* pk = reinterpret_cast<uint32_t*>(&uk);
            uint32_t* pv = reinterpret_cast<uint32_t*>(&uv);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int idx = q4 * 8 + e * 2;
              pk[e] = pack_bf16x2(__uint_as_float(rk[idx]) * p.scale, __uint_as_float(rk[idx + 1]) * p.scale);
              pv[e] = pack_bf16x2(__uint_as_float(rv[idx]), __uint_as_float(rv[idx + 1]));
            }
            *reinterpret_cast<uint4*>(dkr + c * 32 + q4 * 8) = uk;
            *reinterpret_cast<uint4*>(dvr + c * 32 + q4 * 8) = uv;
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

// Row statistics and the cleared dQ accumulator in one pass: ndelta[b, h, s] = -sum_d O dO, nlse2 = -lse * log2(e).
// Bound by memory; HD / 8 lanes share a row with one 16-byte load of O and dO each, a thread takes four rows at once.
// WIDE = false: rows on 8-byte boundaries only (a caller's own pitch), two loads for one.
constexpr int P3_ROWS = 4;
template <bool WIDE>
__device__ __forceinline__ uint4 load_8_bf16(const __nv_bfloat16* p) {
  if constexpr (WIDE) return *reinterpret_cast<const uint4*>(p);
  const uint2 a = reinterpret_cast<const uint2*>(p)[0], b = reinterpret_cast<const uint2*>(p)[1];
  return make_uint4(a.x, a.y, b.x, b.y);
}
template <int HD, bool WIDE>
__global__ void __launch_bounds__(256)
attn_bwd_prep3_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                      const float* __restrict__ lse, float* __restrict__ ndelta, float* __restrict__ nlse2,
                      float* __restrict__ dq_acc, int S, int Hq, long long ldo, long long lddo) {
  constexpr int LPR = HD / 8, RPB = 256 / LPR;
  const int l = threadIdx.x % LPR;
  const int s0 = blockIdx.x * (RPB * P3_ROWS) + threadIdx.x / LPR;
  const int h = blockIdx.y, b = blockIdx.z;
  const long long hb = ((long long)b * Hq + h) * S;
  uint4 a[P3_ROWS], g[P3_ROWS];
#pragma unroll
  for (int k = 0; k < P3_ROWS; ++k) {
    const int s = s0 + k * RPB;
    if (s < S) {
      const long long t = (long long)b * S + s;
      a[k] = load_8_bf16<WIDE>(o + t * ldo + h * HD + l * 8);
      g[k] = load_8_bf16<WIDE>(dout + t * lddo + h * HD + l * 8);
    }
  }
#pragma unroll
  for (int k = 0; k < P3_ROWS; ++k) {
    const int s = s0 + k * RPB;
    float acc = 0.f;
    if (s < S) {
      const uint32_t* x = reinterpret_cast<const uint32_t*>(&a[k]);
      const uint32_t* y = reinterpret_cast<const uint32_t*>(&g[k]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 u = unpack_bf16x2(x[q]), w = unpack_bf16x2(y[q]);
        acc += u.x * w.x + u.y * w.y;
      }
    }
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (s < S) {
      float4* z = reinterpret_cast<float4*>(dq_acc + (hb + s) * HD + l * 8);
      z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (l == 0) {
        ndelta[hb + s] = -acc;
        nlse2[hb + s] = -lse[hb + s] * 1.4426950408889634f;
      }
    }
  }
}

// dq[b * S + s, h * HD + d] = bf16(scale * acc[b, h, s, d]); eight elements to a thread and row, four rows at once.
template <int HD, bool WIDE>
__global__ void __launch_bounds__(256)
dq_rows_to_bf16_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, int S, int Hq, long long lddq,
                       float scale) {
  constexpr int LPR = HD / 8, RPB = 256 / LPR;
  const int l = threadIdx.x % LPR;
  const int s0 = blockIdx.x * (RPB * P3_ROWS) + threadIdx.x / LPR;
  const int h = blockIdx.y, b = blockIdx.z;
  const long long hb = ((long long)b * Hq + h) * S;
  float4 f[P3_ROWS][2];
#pragma unroll
  for (int k = 0; k < P3_ROWS; ++k) {
    const int s = s0 + k * RPB;
    if (s < S) {
      const float4* x = reinterpret_cast<const float4*>(acc + (hb + s) * HD + l * 8);
      f[k][0] = x[0];
      f[k][1] = x[1];
    }
  }
#pragma unroll
  for (int k = 0; k < P3_ROWS; ++k) {
    const int s = s0 + k * RPB;
    if (s < S) {
      uint4 u;
      u.x = pack_bf16x2(f[k][0].x * scale, f[k][0].y * scale);
      u.y = pack_bf16x2(f[k][0].z * scale, f[k][0].w * scale);
      u.z = pack_bf16x2(f[k][1].x * scale, f[k][1].y * scale);
      u.w = pack_bf16x2(f[k][1].z * scale, f[k][1].w * scale);
      __nv_bfloat16* out = dq + ((long long)b * S + s) * lddq + (long long)h * HD + l * 8;
      if constexpr (WIDE) {
        *reinterpret_cast<uint4*>(out) = u;
      } else {
        reinterpret_cast<uint2*>(out)[0] = make_uint2(u.x, u.y);
        reinterpret_cast<uint2*>(out)[1] = make_uint2(u.z, u.w);
      }
    }
  }
}

template <int HD>
static int launch_fa_bwd3(const void* q, const void* k, const void* v, const void* dout, long long ldq, long long ldk,
                          long long ldv, long long lddo, FaBwd3Params& p, cudaStream_t stream) {
  using Cfg = FaBwd3Cfg<HD>;
  static gf::DeviceOnce configured;
  auto kern = fa_bwd3_kernel<HD>;
  if (configured.todo()) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess)
      return GFH_CUDA;
    configured.mark();
  }
  const uint64_t T = (uint64_t)p.B * p.S;
  CUtensorMap tq, tk, tv, tdo;
  int rc = make_tmap_2d(&tq, q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, (uint64_t)p.Hq * HD, ldq * 2, B3_TILE, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tdo, dout, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, (uint64_t)p.Hq * HD, lddo * 2, B3_TILE, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tk, k, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, (uint64_t)p.Hkv * HD, ldk * 2, B3_TILE, 64);
  if (rc) return rc;
  rc = make_tmap_2d(&tv, v, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, T, (uint64_t)p.Hkv * HD, ldv * 2, B3_TILE, 64);
  if (rc) return rc;
  dim3 grid(p.Hkv * p.B, p.S / B3_TILE);
  kern<<<grid, B3_THREADS, Cfg::SMEM_BYTES, stream>>>(tq, tk, tv, tdo, p);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

}  // namespace gf

using namespace gf;

// ndelta, nlse2: fp32 [B, Hq, S]; dq_acc: fp32 [B, Hq, S, HD], cleared. Rows of o and dout on 8-byte boundaries.
GF_API int gf_attn_bwd_prep3(const void* o, const void* dout, const float* lse, float* ndelta, float* nlse2,
                             float* dq_acc, int B, int S, int Hq, int HD, long long ldo, long long lddo, void* stream) {
  gf::enter();
  if (B <= 0 || S <= 0 || Hq <= 0 || B > 65535 || Hq > 65535 || (ldo % 4) || (lddo % 4) || (HD != 64 && HD != 128) ||
      ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout)) & 7) || (reinterpret_cast<uintptr_t>(dq_acc) & 15))
    return GFH_BAD_ARG;
  const bool wide = ldo % 8 == 0 && lddo % 8 == 0 &&
                    ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout)) & 15) == 0;
  const int rows = 256 / (HD / 8) * P3_ROWS;
  const dim3 grid((S + rows - 1) / rows, Hq, B);
  auto kern = HD == 128 ? (wide ? attn_bwd_prep3_kernel<128, true> : attn_bwd_prep3_kernel<128, false>)
                        : (wide ? attn_bwd_prep3_kernel<64, true> : attn_bwd_prep3_kernel<64, false>);
  kern<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)dout, lse, ndelta, nlse2,
                                               dq_acc, S, Hq, ldo, lddo);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// Statistics and accumulator as gf_attn_bwd_prep3 leaves them; the accumulator receives dQ / scale, so convert afterwards
// with gf_dq_rows_to_bf16(..., scale). S must be a multiple of 128.
GF_API int gf_flash_attn_bwd3(const void* q, const void* k, const void* v, const void* dout, const float* nlse2,
                              const float* ndelta, float* dq_acc, void* dk, void* dv, int B, int S, int Hq, int Hkv,
                              int head_dim, long long ldq, long long ldk, long long ldv, long long lddo,
                              long long lddk, long long lddv, float scale, int causal, int* status, void* stream) {
  gf::enter();
  if (B <= 0 || S <= 0 || (S % B3_TILE) || Hq <= 0 || Hkv <= 0 || Hq % Hkv) return GFH_BAD_ARG;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (lddo % 8) || (lddk % 8) || (lddv % 8)) return GFH_BAD_ARG;
  if (((reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv) | reinterpret_cast<uintptr_t>(nlse2) |
        reinterpret_cast<uintptr_t>(ndelta) | reinterpret_cast<uintptr_t>(dq_acc)) & 15) || S / B3_TILE > 65535)
    return GFH_BAD_ARG;
  FaBwd3Params p;
  p.B = B; p.S = S; p.Hq = Hq; p.Hkv = Hkv; p.causal = causal; p.scale = scale;
  p.nlse2 = nlse2; p.ndelta = ndelta; p.dq_acc = dq_acc;
  p.dK = (__nv_bfloat16*)dk; p.lddk = lddk; p.dV = (__nv_bfloat16*)dv; p.lddv = lddv; p.status = status;
  p.head_group = attention_head_group_l2(B * Hkv, 4ll * S * head_dim * (Hq / Hkv));
  if (head_dim == 128) return launch_fa_bwd3<128>(q, k, v, dout, ldq, ldk, ldv, lddo, p, (cudaStream_t)stream);
  if (head_dim == 64) return launch_fa_bwd3<64>(q, k, v, dout, ldq, ldk, ldv, lddo, p, (cudaStream_t)stream);
  return GFH_BAD_ARG;
}

// Converts the fp32 dQ accumulator [B, Hq, S, HD] into bf16 rows with pitch lddq, on 8-byte boundaries.
GF_API int gf_dq_rows_to_bf16(const float* acc, void* dq, int B, int S, int Hq, int HD, long long lddq, float scale,
                              void* stream) {
  gf::enter();
  if (B <= 0 || S <= 0 || Hq <= 0 || B > 65535 || Hq > 65535 || (lddq % 4) || (HD != 64 && HD != 128) ||
      (reinterpret_cast<uintptr_t>(acc) & 15) || (reinterpret_cast<uintptr_t>(dq) & 7))
    return GFH_BAD_ARG;
  const bool wide = lddq % 8 == 0 && (reinterpret_cast<uintptr_t>(dq) & 15) == 0;
  const int rows = 256 / (HD / 8) * P3_ROWS;
  const dim3 grid((S + rows - 1) / rows, Hq, B);
  auto kern = HD == 128 ? (wide ? dq_rows_to_bf16_kernel<128, true> : dq_rows_to_bf16_kernel<128, false>)
                        : (wide ? dq_rows_to_bf16_kernel<64, true> : dq_rows_to_bf16_kernel<64, false>);
  kern<<<grid, 256, 0, (cudaStream_t)stream>>>(acc, (__nv_bfloat16*)dq, S, Hq, lddq, scale);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}
