// A pre-norm transformer block (GPT-2: LayerNorm, biases, GELU), forward and backward pass, each in one call:
//
//   h = x + Wo attention(LN1(x) Wqkv^T + bqkv) + bo        y = h + W2 gelu(LN2(h) W1^T + b1) + b2
//
// Host code only: the launches are those of the layers one by one, in the same order with the same operands, so results are the
// same bits, with two exceptions: the sums of a gradient with the one that arrives past the branch are taken inside the
// LayerNorm backward kernels (rounded once instead of twice), and products whose parts of K are added with atomics (few tiles
// and a long K, see gemm_bf16.cu) differ from call to call as they do in the layers. From Python the layers' 38 launches kept
// the host busy for 1000 to 1200 us where the device had work for 780 (8192 tokens of width 768).
#include <math.h>

#include <algorithm>

#include "gf_host.h"

GF_API int gf_layernorm_fwd(const void* x, const void* w, const void* b, void* y, float* mean, float* rstd, int T, int D, float eps,
                            void* stream);
GF_API int gf_layernorm_bwd_res(const void* x, const void* w, const void* dy, const float* mean, const float* rstd, const void* dres,
                                void* dx, void* dw, void* db, float* scratch, int T, int D, int accumulate, void* stream);
GF_API int gf_norm_bwd_grid(int T);
GF_API int gf_colsum_bf16(const void* x, long long ld, void* out, float* scratch, int T, int D, int accumulate, void* stream);
GF_API int gf_unary_fwd(const void* x, void* y, long long n, int op, int dtype, void* stream);
GF_API int gf_unary_bwd_bf16(const void* x, const void* dy, void* dx, long long n, int op, void* stream);
GF_API long long gf_gemm_bf16_workspace(int M, int N, int K, int a_mn_major, int b_mn_major, int aligned, int out_fp32, int accumulate,
                                        int activation);
GF_API int gf_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, int a_mn_major, long long lda, int b_mn_major,
                        long long ldb, long long ldc, int out_fp32, int accumulate, const void* bias, const void* residual,
                        long long ldr, float alpha, int* status, int bn_hint, int max_ctas, const int* splitk_ws, int activation,
                        int splitk_ws_floats, void* stream);
GF_API int gf_flash_attn_fwd3(const void* q, const void* k, const void* v, void* o, float* lse, int B, int S, int Hq, int Hkv,
                              int head_dim, long long ldq, long long ldk, long long ldv, long long ldo, float scale, int causal,
                              int* status, void* stream);
GF_API int gf_attn_bwd_prep3(const void* o, const void* dout, const float* lse, float* ndelta, float* nlse2, float* dq_acc, int B,
                             int S, int Hq, int HD, long long ldo, long long lddo, void* stream);
GF_API int gf_flash_attn_bwd3(const void* q, const void* k, const void* v, const void* dout, const float* nlse2, const float* ndelta,
                              float* dq_acc, void* dk, void* dv, int B, int S, int Hq, int Hkv, int head_dim, long long ldq,
                              long long ldk, long long ldv, long long lddo, long long lddk, long long lddv, float scale, int causal,
                              int* status, void* stream);
GF_API int gf_dq_rows_to_bf16(const float* acc, void* dq, int B, int S, int Hq, int HD, long long lddq, float scale, void* stream);

namespace gf {
namespace {

constexpr int ACT_GELU = 1;

struct Carve {                       // pieces of a buffer on 256-byte boundaries; with a null base only their sum
  uint8_t* base;
  long long used = 0;
  void* take(long long bytes) {
    void* r = base ? base + used : nullptr;
    used += (bytes + 255) & ~255ll;
    return r;
  }
};

struct Block {
  int B, S, E, F, H, Hk, D, T, P;    // tokens; width of the packed projection
  Block(int B_, int S_, int E_, int F_, int H_, int Hk_) : B(B_), S(S_), E(E_), F(F_), H(H_), Hk(Hk_) {
    D = H > 0 ? E / H : 0;
    T = B * S;
    P = (H + 2 * Hk) * D;
  }
  bool ok() const {
    return B > 0 && S > 0 && E > 0 && F > 0 && H > 0 && Hk > 0 && H % Hk == 0 && H * D == E && (D == 64 || D == 128) && E % 8 == 0 &&
           F % 8 == 0 && (long long)B * S <= 0x7fffffffll / 8;
  }
};

// fp32 values a product takes as workspace
long long product_floats(int M, int N, int K, int a_mn_major, int b_mn_major) {
  return gf_gemm_bf16_workspace(M, N, K, a_mn_major, b_mn_major, 1, 0, 0, 0);
}
// The most that the products y = x W^T of the forward pass take, and the two gradients of one of them, W [N, K].
long long forward_floats(const Block& b) {
  return std::max({product_floats(b.T, b.P, b.E, 0, 0), product_floats(b.T, b.E, b.E, 0, 0), product_floats(b.T, b.F, b.E, 0, 0),
                   product_floats(b.T, b.E, b.F, 0, 0)});
}
long long gradient_floats(const Block& b, int N, int K) {
  return std::max(product_floats(b.T, K, N, 0, 1), product_floats(N, K, b.T, 1, 1));
}

// Results of the forward pass. With `keep` all of them have a place of their own and the backward pass reads them again.
// Without, only what is still to be read has: n1, o and n2 take turns in y, which is written last; pre follows q, k, v.
struct Results {
  void *n1, *qkv, *o, *h, *n2, *pre, *act;
  float *stats1 = nullptr, *lse = nullptr, *stats2 = nullptr;
  long long bytes;
  Results(const Block& b, bool keep, void* base, void* y) {
    Carve c{(uint8_t*)base};
    if (!keep) {
      n1 = o = n2 = y;
      qkv = pre = c.take(2ll * b.T * std::max(b.P, b.F));
      h = c.take(2ll * b.T * b.E);
      act = c.take(2ll * b.T * b.F);
      bytes = c.used;
      return;
    }
    n1 = c.take(2ll * b.T * b.E);
    stats1 = (float*)c.take(8ll * b.T);
    qkv = c.take(2ll * b.T * b.P);
    o = c.take(2ll * b.T * b.E);
    lse = (float*)c.take(4ll * b.T * b.H);
    h = c.take(2ll * b.T * b.E);
    n2 = c.take(2ll * b.T * b.E);
    stats2 = (float*)c.take(8ll * b.T);
    pre = c.take(2ll * b.T * b.F);
    act = c.take(2ll * b.T * b.F);
    bytes = c.used;
  }
  static constexpr int PARTS = 10;
  void get(const void** p) const {
    const void* all[PARTS] = {n1, stats1, qkv, o, lse, h, n2, stats2, pre, act};
    std::copy(all, all + PARTS, p);
  }
  void set(const void* const* p) {
    n1 = (void*)p[0]; stats1 = (float*)p[1]; qkv = (void*)p[2]; o = (void*)p[3]; lse = (float*)p[4];
    h = (void*)p[5]; n2 = (void*)p[6]; stats2 = (float*)p[7]; pre = (void*)p[8]; act = (void*)p[9];
  }
};

// Temporaries of the backward pass. The gradient of h lives where the one of x is written in the end; the second layer's
// (`wide` and its products' workspace) are done with when the attention's, in the same place, begin.
struct Temps {
  void *wide, *dn, *dqkv;
  float *ndelta, *nlse2, *dq_acc, *sums, *ws_mlp, *ws_out, *ws_qkv;
  long long bytes;
  Temps(const Block& b, void* base) {
    Carve c{(uint8_t*)base};
    dn = c.take(2ll * b.T * b.E);                // of a norm's output, then of the attention output
    ndelta = (float*)c.take(4ll * b.T * b.H);
    nlse2 = (float*)c.take(4ll * b.T * b.H);
    sums = (float*)c.take(4ll * gf_norm_bwd_grid(b.T) * std::max({2 * b.E, b.P, b.F}));
    Carve mlp = c, out = c, att = c;
    wide = mlp.take(2ll * b.T * b.F);            // gradient of the activation, then of its input
    ws_mlp = (float*)mlp.take(4 * std::max(gradient_floats(b, b.F, b.E), gradient_floats(b, b.E, b.F)));
    ws_out = (float*)out.take(4 * gradient_floats(b, b.E, b.E));
    dqkv = att.take(2ll * b.T * b.P);
    const long long ws_bytes = 4 * gradient_floats(b, b.P, b.E), acc_bytes = 4ll * b.T * b.E;
    dq_acc = ws_qkv = (float*)att.take(std::max(acc_bytes, ws_bytes));
    bytes = std::max({mlp.used, out.used, att.used});
  }
};

}  // namespace
}  // namespace gf

// Bytes of the buffer `saved` that the forward pass fills for the backward pass (which = 0), of the backward pass's workspace
// (which = 1), and of the forward pass's with `saved` (which = 2, often none) and without (which = 3). -1: sizes that are not
// taken.
GF_API long long gf_gpt_block_bytes(int which, int B, int S, int E, int F, int H, int Hk) {
  gf::Block b(B, S, E, F, H, Hk);
  if (!b.ok()) return -1;
  if (which == 0) return gf::Results(b, true, nullptr, nullptr).bytes;
  if (which == 1) return gf::Temps(b, nullptr).bytes;
  const long long ws = (4 * gf::forward_floats(b) + 255) & ~255ll;
  return which == 2 ? ws : ws + gf::Results(b, false, nullptr, nullptr).bytes;
}

// Where in `saved` its ten tensors begin (bytes), in the order n1 [T, E], statistics [2, T] fp32, q k v [T, (H + 2 Hk) D], o
// [T, E], lse [B, H, S] fp32, h [T, E], n2 [T, E], statistics [2, T] fp32, pre [T, F], act [T, F].
GF_API int gf_gpt_block_parts(long long* offsets, int B, int S, int E, int F, int H, int Hk) {
  using namespace gf;
  const Block b(B, S, E, F, H, Hk);
  if (!b.ok() || !offsets) return GFH_BAD_ARG;
  uint8_t* base = reinterpret_cast<uint8_t*>(256);         // only differences are taken
  const void* at[Results::PARTS];
  Results(b, true, base, nullptr).get(at);
  for (int i = 0; i < Results::PARTS; ++i) offsets[i] = (const uint8_t*)at[i] - base;
  return GFH_OK;
}

// params: {ln1 weight, bias, Wqkv, bqkv, Wo, bo, ln2 weight, bias, W1, b1, W2, b2}, biases may be null; dense bf16.
// x, y: dense bf16 [B * S, E]. saved: null where there is no backward pass.
// saved_bytes, ws_bytes: what the caller allocated; less than gf_gpt_block_bytes is refused before the first launch.
GF_API int gf_gpt_block_fwd(const void* x, const void* const* params, void* y, void* saved, long long saved_bytes, void* ws,
                            long long ws_bytes, int B, int S, int E, int F, int H, int Hk, int causal, float eps1, float eps2,
                            int* status, void* stream) {
  using namespace gf;
  bind();
  const Block b(B, S, E, F, H, Hk);
  if (!b.ok() || !x || !y) return GFH_BAD_ARG;
  const long long product_bytes = (4 * forward_floats(b) + 255) & ~255ll;
  const Results s(b, saved != nullptr, saved ? saved : (uint8_t*)ws + product_bytes, y);
  if (saved ? saved_bytes < s.bytes || ws_bytes < product_bytes : ws_bytes < product_bytes + s.bytes) return GFH_BAD_ARG;
  const int T = b.T, P = b.P, D = b.D;
  int rc;
  auto linear = [&](const void* in, int K, const void* w, const void* bias, const void* res, void* out, int N) {
    const long long fl = product_floats(T, N, K, 0, 0);
    return gf_gemm_bf16(in, w, out, T, N, K, 0, K, 0, K, N, 0, 0, bias, res, res ? N : 0, 1.f, status, 0, 0,
                        fl ? (const int*)ws : nullptr, 0, (int)fl, stream);
  };
  if ((rc = gf_layernorm_fwd(x, params[0], params[1], s.n1, s.stats1, s.stats1 ? s.stats1 + T : nullptr, T, E, eps1, stream))) return rc;
  if ((rc = linear(s.n1, E, params[2], params[3], nullptr, s.qkv, P))) return rc;
  const uint8_t* q = (const uint8_t*)s.qkv;
  if ((rc = gf_flash_attn_fwd3(q, q + 2ll * E, q + 2ll * (E + Hk * D), s.o, s.lse, B, S, H, Hk, D, P, P, P, E,
                               1.f / sqrtf((float)D), causal, status, stream)))
    return rc;
  if ((rc = linear(s.o, E, params[4], params[5], x, s.h, E))) return rc;
  if ((rc = gf_layernorm_fwd(s.h, params[6], params[7], s.n2, s.stats2, s.stats2 ? s.stats2 + T : nullptr, T, E, eps2, stream)))
    return rc;
  if ((rc = linear(s.n2, E, params[8], params[9], nullptr, s.pre, F))) return rc;
  if ((rc = gf_unary_fwd(s.pre, s.act, (long long)T * F, ACT_GELU, 1, stream))) return rc;
  return linear(s.act, F, params[10], params[11], s.h, y, E);
}

// grads: where the gradients of params go, null for those that are not wanted; the norms' are always written. dx likewise.
// saved: as the forward pass left it, or null and `parts`: its ten tensors one by one, where something moved them in between.
// ws: gf_gpt_block_bytes(1, ...) bytes; the sizes of both buffers are checked as above. S must be a multiple of 128.
GF_API int gf_gpt_block_bwd(const void* x, const void* const* params, const void* dy, const void* saved, long long saved_bytes,
                            const void* const* parts, void* dx, void* const* grads, void* ws, long long ws_bytes, int B, int S, int E, int F, int H, int Hk,
                            int causal, int* status, void* stream) {
  using namespace gf;
  bind();
  const Block b(B, S, E, F, H, Hk);
  if (!b.ok() || !x || !dy || (!saved && !parts) || !ws || !dx || !grads || !grads[0] || !grads[6] || S % 128) return GFH_BAD_ARG;
  Results s(b, true, const_cast<void*>(saved), nullptr);
  const Temps t(b, ws);
  if ((saved && saved_bytes < s.bytes) || ws_bytes < t.bytes) return GFH_BAD_ARG;
  if (!saved) s.set(parts);
  const int T = b.T, P = b.P, D = b.D;
  const float scale = 1.f / sqrtf((float)D);
  int rc;
  // gradients of y = in W^T + bias at dy [T, N]: of in (to `din`), W and bias
  auto linear = [&](const void* g, int N, const void* in, int K, const void* w, void* din, void* dw, void* db, float* ws_at) {
    auto product = [&](const void* A, int a_mn, int lda, const void* W, int ldw, void* out, int m, int n, int k) {
      const long long fl = product_floats(m, n, k, a_mn, 1);
      return gf_gemm_bf16(A, W, out, m, n, k, a_mn, lda, 1, ldw, n, 0, 0, nullptr, nullptr, 0, 1.f, status, 0, 0,
                          fl ? (const int*)ws_at : nullptr, 0, (int)fl, stream);
    };
    if ((rc = product(g, 0, N, w, K, din, T, K, N))) return rc;
    if (dw && (rc = product(g, 1, N, in, K, dw, N, K, T))) return rc;
    if (db) rc = gf_colsum_bf16(g, N, db, t.sums, T, N, 0, stream);
    return rc;
  };
  void* dh = dx;                     // of h: until the last launch, which reads it where it writes dx
  if (linear(dy, E, s.act, F, params[10], t.wide, grads[10], grads[11], t.ws_mlp)) return rc;
  if ((rc = gf_unary_bwd_bf16(s.pre, t.wide, t.wide, (long long)T * F, ACT_GELU, stream))) return rc;
  if (linear(t.wide, F, s.n2, E, params[8], t.dn, grads[8], grads[9], t.ws_mlp)) return rc;
  if ((rc = gf_layernorm_bwd_res(s.h, params[6], t.dn, s.stats2, s.stats2 + T, dy, dh, grads[6], grads[7], t.sums, T, E, 0, stream)))
    return rc;
  if (linear(dh, E, s.o, E, params[4], t.dn, grads[4], grads[5], t.ws_out)) return rc;
  const uint8_t* q = (const uint8_t*)s.qkv;
  uint8_t* dq = (uint8_t*)t.dqkv;
  const long long ok = 2ll * E, ov = 2ll * (E + Hk * D);
  if ((rc = gf_attn_bwd_prep3(s.o, t.dn, s.lse, t.ndelta, t.nlse2, t.dq_acc, B, S, H, D, E, E, stream))) return rc;
  if ((rc = gf_flash_attn_bwd3(q, q + ok, q + ov, t.dn, t.nlse2, t.ndelta, t.dq_acc, dq + ok, dq + ov, B, S, H, Hk, D, P, P, P, E, P, P,
                               scale, causal, status, stream)))
    return rc;
  if ((rc = gf_dq_rows_to_bf16(t.dq_acc, dq, B, S, H, D, P, scale, stream))) return rc;
  if (linear(t.dqkv, P, s.n1, E, params[2], t.dn, grads[2], grads[3], t.ws_qkv)) return rc;
  return gf_layernorm_bwd_res(x, params[0], t.dn, s.stats1, s.stats1 + T, dh, dx, grads[0], grads[1], t.sums, T, E, 0, stream);
}

// The three launches of the attention backward pass; ws: fp32, B Hq S (D + 2) values on a 16-byte boundary (accumulator first).
// ld: row pitches of q, k, v, o, do, dq, dk, dv.
GF_API int gf_flash_attn_backward(const void* q, const void* k, const void* v, const void* o, const void* dout, const float* lse,
                                  void* dq, void* dk, void* dv, float* ws, int B, int S, int Hq, int Hkv, int D, const long long* ld,
                                  float scale, int causal, int* status, void* stream) {
  gf::bind();
  if (B <= 0 || S <= 0 || Hq <= 0 || S % 128 || !ws) return gf::GFH_BAD_ARG;
  const long long rows = (long long)B * Hq * S;
  float *acc = ws, *ndelta = ws + rows * D, *nlse2 = ndelta + rows;
  int rc = gf_attn_bwd_prep3(o, dout, lse, ndelta, nlse2, acc, B, S, Hq, D, ld[3], ld[4], stream);
  if (rc) return rc;
  rc = gf_flash_attn_bwd3(q, k, v, dout, nlse2, ndelta, acc, dk, dv, B, S, Hq, Hkv, D, ld[0], ld[1], ld[2], ld[4], ld[6], ld[7], scale,
                          causal, status, stream);
  if (rc) return rc;
  return gf_dq_rows_to_bf16(acc, dq, B, S, Hq, D, ld[5], scale, stream);
}
