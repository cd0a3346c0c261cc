// One LLaMA decoder layer for one new token of each sequence: seven kernels from one call (nine with more than 16 sequences;
// one less where the attention needs no merge).
//
//   q, k, v   = rms_norm(x) Wqkv^T                 gemm_rows.cu, the norm in front of the product
//   attention over the caches, rotation of q and k, and the new cache row (attn_decode.cu), and its merge
//   h         = x + attention Wo^T
//   gate, up  = rms_norm(h) Wgu^T
//   a         = silu(gate) * up                    pointwise.cu
//   y         = h + a Wdown^T
//
// The first launch is an ordinary one, so all earlier work of the stream is complete when it runs. Every further kernel may
// start while the one in front of it ends (programmatic stream serialization; the norms of more than 16 sequences do not) and
// fetches what no kernel of the layer writes, weights and older cache rows, before it waits for that one. Each kernel waits for
// the one in front of it before it ends, so a kernel that has waited may read the results of all earlier ones.
//
// Device time in a graph, us, nine ordinary launches of the layers / here: LLaMA-7B (hidden 4096, inner 11008, 32 heads), one
// sequence of 1500 keys 104 / 88, 8 145 / 111, 16 of 300 140 / 96, 32 of 800 207 / 167, 64 of 300 200 / 168; 70B (8192, 28672,
// 64 / 8 heads), one of 1500 283 / 282, 16 of 300 366 / 289; hidden 1024, one of 100 26.3 / 23.7, and 256 18.1 / 21.6, where
// the products' fixed cost is all there is; enqueueing it takes the host 60 us instead of 205. SwiGLU inside the last product,
// computed by every CTA for its part of K, costs more than the kernel and its launch: 88 -> 96 us for one sequence of the
// first, 282 -> 329 of the second. What is left above the bytes (93 us at 8): each kernel ends before the next one's tokens can
// be read, and the memory waits for about 4 us then.
#include <math.h>

#include "gemm_rows.cuh"
#include "gf_host.h"

namespace gf {
int attn_decode_append(const void* qkv, long long ldq, void* kcache, void* vcache, int s_max, int len, const float* cos_row,
                       const float* sin_row, int interleaved, void* out, long long ldo, int B, int Hq, int Hkv, int D, float scale,
                       int splits, float* scratch, int chained, cudaStream_t st);
int swiglu_chained(const void* gu, void* y, long long T, int F, cudaStream_t st);
}
GF_API int gf_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* h_out, float* rstd, int T, int D, float eps,
                          void* stream);

// x, y dense bf16 [B, hidden], dense weights [out, in], caches [B, s_max, Hkv, D], tables [positions, D / 2].
// ws: 256-byte aligned, 2 B ((2 Hq + 2 Hkv) D + hidden + 2 inner + max(hidden, inner)) + 4 B Hq splits (D + 2) + 1536
// bytes.
GF_API int gf_llama_decode_layer(const void* x, const void* attn_norm, float attn_eps, const void* wqkv,
                                 const void* wo, const void* ffn_norm, float ffn_eps, const void* gate_up, const void* down,
                                 const float* cos_t, const float* sin_t, void* kcache, void* vcache, int s_max, void* y, void* ws,
                                 int B, int hidden, int inner, int Hq, int Hkv, int D, int interleaved, int pos, int splits,
                                 int* status, void* stream) {
  using namespace gf;
  bind();
  if (B < 1 || B > ROWS_MAX_M || hidden <= 0 || inner <= 0 || Hq <= 0 || Hkv <= 0 || pos < 0 || pos >= s_max || splits < 1 ||
      !ws || (reinterpret_cast<uintptr_t>(ws) & 255))
    return GFH_BAD_ARG;
  // all that the kernels check or read as 16-byte vectors, before the first of them writes anything
  if ((D != 64 && D != 128) || Hq % Hkv || hidden % 8 || inner % 8) return GFH_BAD_ARG;
  for (const void* p : {x, attn_norm, wqkv, wo, ffn_norm, gate_up, down, (const void*)kcache, (const void*)vcache, (const void*)y})
    if (!p || (reinterpret_cast<uintptr_t>(p) & 15)) return GFH_BAD_ARG;
  if (!cos_t || !sin_t) return GFH_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int att = Hq * D, packed = (Hq + 2 * Hkv) * D;
  uint8_t* at = reinterpret_cast<uint8_t*>(ws);
  auto take = [&](long long bytes) {
    uint8_t* r = at;
    at += (bytes + 255) & ~255ll;
    return r;
  };
  void* qkv = take(2ll * B * packed);
  void* o = take(2ll * B * att);
  void* h = take(2ll * B * hidden);
  void* gu = take(4ll * B * inner);
  void* tmp = take(2ll * B * (hidden > inner ? hidden : inner));
  float* parts = reinterpret_cast<float*>(take(4ll * B * Hq * splits * (D + 2)));
  const long long half = (long long)pos * (D / 2);

  // Up to 16 rows the norms run in front of the products that read them. With more, every CTA would compute more of them than
  // it has time for beside its weights, and they are kernels of their own.
  const bool fused = B <= ROWS_MAX_M_FUSED;
  int rc = GFH_OK;
  auto normed_gemm = [&](const void* in, long long ld, const void* w_norm, float eps, const void* w, void* out, int n, int chained) {
    RowsGemm g{in, ld, w, hidden, out, n, 0, B, n, hidden, ROWS_RMSNORM, w_norm, eps, nullptr, nullptr, 0, 1.f, 0, status};
    if (!fused) {
      if ((rc = gf_rmsnorm_fwd(in, nullptr, w_norm, tmp, nullptr, nullptr, B, hidden, eps, st))) return rc;
      g.X = tmp; g.ldx = hidden; g.input = ROWS_PLAIN;
      chained = 1;
    }
    return rc = gemm_rows_run(g, chained, st);
  };
  if (normed_gemm(x, hidden, attn_norm, attn_eps, wqkv, qkv, packed, 0)) return rc;
  if ((rc = attn_decode_append(qkv, packed, kcache, vcache, s_max, pos + 1, cos_t + half, sin_t + half, interleaved, o, att, B, Hq,
                               Hkv, D, 1.f / sqrtf((float)D), splits, parts, 1, st)))
    return rc;
  RowsGemm g{o, att, wo, att, h, hidden, 0, B, hidden, att, ROWS_PLAIN, nullptr, 0.f, nullptr, x, hidden, 1.f, 0, status};
  if ((rc = gemm_rows_run(g, 1, st))) return rc;
  if (normed_gemm(h, hidden, ffn_norm, ffn_eps, gate_up, gu, 2 * inner, 1)) return rc;
  if ((rc = swiglu_chained(gu, tmp, B, inner, st))) return rc;
  g = RowsGemm{tmp, inner, down, inner, y, hidden, 0, B, hidden, inner, ROWS_PLAIN, nullptr, 0.f, nullptr, h, hidden, 1.f, 0, status};
  rc = gemm_rows_run(g, 1, st);
  note_extra_launches(5);                    // four products and the attention; its merge, norms and SwiGLU are counted where they start
  return rc;
}
