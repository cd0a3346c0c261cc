// Softmax cross-entropy (fused forward + gradient, logits read from HBM once) and the
// flat fused AdamW / Adam / SGD updates on fp32 master weights with a bf16 copy-out.
//
// Cross-entropy: mean over rows of -log_softmax(logits)[target]
// (ghostflow-nn/src/loss.rs:75-103; gradient softmax - onehot, ghostflow-autograd/src/backward.rs:171-191).
// AdamW: p*(1 - lr*wd) - lr * mhat / (sqrt(vhat) + eps), m and v from the raw gradient
// (ghostflow-optim/src/adam.rs:162-197); Adam with L2-coupled decay (adam.rs:52-95);
// SGD with momentum/dampening/nesterov (ghostflow-optim/src/sgd.rs:54-93).
#include "gf_host.h"
#include "gf_ptx.cuh"

#include <algorithm>
#include <new>

namespace gf {

// One CTA of 256 threads per row, as many on an SM as have room for their row in shared memory, each walking its rows: a bulk
// copy brings the row, the threads take maximum and sum in one reduction (every thread sums against its own maximum and
// the pairs are merged) and write the gradient, and the next copy starts. Loads, exponentials (two per logit, a third of
// the time by themselves) and stores of one CTA follow one another; it is the CTAs of an SM, each in another phase, that
// keep memory and special-function unit busy together. So small CTAs win, with no more registers than six of them
// have, and the arithmetic goes two logits to an instruction.
// dlogits overwrite the logits in place or go to a separate buffer. loss_rows[t] = logsumexp - x[target]; ignored rows give 0.
// Measured, before (512 threads per row, plain loads, three reductions) -> now: [8192, 50257] 438 -> 306 us (5.4 TB/s),
// [8192, 30522] 258 -> 179, [4096, 32000] 138 -> 98, [8192, 16384] 145 -> 95, [8192, 8192] 85 -> 59, [8192, 1000] 34 -> 25.
// Others tried at [8192, 50257] / [8192, 30522]: 512 threads 304 / 184, 1024 threads 330 / 235, one CTA of 1024 with a ring of
// rows and the row in registers 362 / 214, a quarter of the exponentials by polynomial 396 / 220.
constexpr int XENT_THREADS = 256;
constexpr int XENT_CTAS = 6;
constexpr size_t XENT_SMEM = 220 * 1024;    // of an SM, for rows

// e^(x + nm) of a packed pair of logits, as 2^((x + nm) log2 e) on the ex2 instruction
__device__ __forceinline__ uint64_t exp_two(uint32_t bf16_pair, uint64_t nm) {
  const uint64_t x = pk2f(__uint_as_float(bf16_pair << 16), __uint_as_float(bf16_pair & 0xffff0000u));
  const uint64_t y = f2_mul(f2_add(x, nm), pk2f(1.4426950408889634f, 1.4426950408889634f));
  return pk2f(ex2_approx(lo2(y)), ex2_approx(hi2(y)));
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {     // a NaN leaves the other operand
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// Over the warp: m becomes the maximum M, s the sum of s e^(m - M). A part without a finite maximum has sum 0.
__device__ __forceinline__ void warp_max_sum(float& m, float& s) {
  const float own = m;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(m) : "f"(own));   // a NaN is passed over, as by fmaxf
  s *= own == m ? 1.f : __expf(own - m);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
}

__global__ void __launch_bounds__(XENT_THREADS, XENT_CTAS)
xent_kernel(const __nv_bfloat16* logits, const long long* __restrict__ targets, float* __restrict__ loss_rows,
                 __nv_bfloat16* dlogits, int T, int V, long long ld, float grad_scale, long long ignore_index, int* status) {
  extern __shared__ __align__(128) uint8_t rowbuf[];
  __shared__ uint64_t full;
  __shared__ float red[2][2][32];     // of alternate rows: maximum and sum of every warp
  const int nv = (V + 7) >> 3;
  const uint32_t row_bytes = (uint32_t)nv * 16;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 32) {               // warps that there are not add nothing
    red[0][0][threadIdx.x] = red[1][0][threadIdx.x] = -INFINITY;
    red[0][1][threadIdx.x] = red[1][1][threadIdx.x] = 0.f;
  }
  if (threadIdx.x == 0) {
    mbar_init(&full, 1);
    mbar_fence_init();
  }
  __syncthreads();
  auto load = [&](long long row) {
    mbar_expect_tx(&full, row_bytes);
    bulk_load_1d(rowbuf, logits + row * ld, row_bytes, &full);
  };
  if (threadIdx.x == 0 && blockIdx.x < T) load(blockIdx.x);
  uint4* xs = reinterpret_cast<uint4*>(rowbuf);
  int k = 0;
  for (long long row = blockIdx.x; row < T; row += gridDim.x, ++k) {
    const long long tgt = targets[row];
    const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= V;
    const bool ok = mbar_wait(&full, k & 1);
    constexpr uint32_t NONE = 0xFF80FF80u;     // bf16 -inf twice: adds nothing to the sum and gets gradient 0
    uint32_t mp = NONE;
    for (int v = threadIdx.x; v < nv; v += XENT_THREADS) {
      uint4 u = xs[v];
      // The host guarantees ld % 8 == 0 and ld >= round_up(V, 8): the last vector lies inside the row's pitch, and those
      // of its columns that are behind the row do not count.
      if (v == nv - 1) {
        const int c = V - v * 8;
        uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = 2 * q >= c ? NONE : 2 * q + 1 >= c ? (w[q] & 0xffffu) | (NONE & 0xffff0000u) : w[q];
        u = make_uint4(w[0], w[1], w[2], w[3]);
        xs[v] = u;
      }
      mp = max_bf16x2(max_bf16x2(mp, max_bf16x2(u.x, u.y)), max_bf16x2(u.z, u.w));
    }
    const float2 m2 = unpack_bf16x2(mp);
    float m = fmaxf(m2.x, m2.y);
    const float m0 = m == -INFINITY ? 0.f : -m;
    const uint64_t nm0 = pk2f(m0, m0);
    uint64_t sa = 0, sb = 0;
#pragma unroll 2
    for (int v = threadIdx.x; v < nv; v += XENT_THREADS) {
      const uint4 u = xs[v];
      sa = f2_add(sa, exp_two(u.x, nm0));
      sb = f2_add(sb, exp_two(u.y, nm0));
      sa = f2_add(sa, exp_two(u.z, nm0));
      sb = f2_add(sb, exp_two(u.w, nm0));
    }
    sa = f2_add(sa, sb);
    float s = lo2(sa) + hi2(sa);
    warp_max_sum(m, s);
    if (lane == 0) {
      red[k & 1][0][warp] = m;
      red[k & 1][1][warp] = s;
    }
    if (!__syncthreads_and(ok)) {              // the copy never arrived: all threads give up together
      if (threadIdx.x == 0) atomicCAS(status, 0, GF_ERR_WAIT_FULL);
      error_drain_pause();
      break;
    }
    m = red[k & 1][0][lane];
    s = red[k & 1][1][lane];
    warp_max_sum(m, s);
    if (m == -INFINITY) s = __int_as_float(0x7fffffff);    // no finite logit in the row: no probabilities either
    if (threadIdx.x == 0)
      loss_rows[row] = ignored ? 0.f : logf(s) + m - __bfloat162float(reinterpret_cast<__nv_bfloat16*>(rowbuf)[tgt]);
    if (dlogits) {
      const float inv = ignored ? 0.f : grad_scale / s;
      uint4* dr = reinterpret_cast<uint4*>(dlogits + row * ld);
      const int tv = ignored ? -1 : (int)(tgt >> 3), tj = (int)(tgt & 7);
      const uint64_t nm = pk2f(-m, -m), inv2 = pk2f(inv, inv);
#pragma unroll 2
      for (int v = threadIdx.x; v < nv; v += XENT_THREADS) {
        const uint4 u = xs[v];
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
        uint32_t o[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint64_t g = f2_mul(exp_two(w[q], nm), inv2);
          float g0 = lo2(g), g1 = hi2(g);
          if (v == tv) {
            g0 -= 2 * q == tj ? grad_scale : 0.f;
            g1 -= 2 * q + 1 == tj ? grad_scale : 0.f;
          }
          o[q] = pack_bf16x2(g0, g1);
        }
        dr[v] = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0 && row + gridDim.x < T) load(row + gridDim.x);
  }
}

// ------------------------------------------------------------------ flat optimizers
struct AdamArgs {
  float lr, beta1, beta2, eps, wd, bc1, bc2, grad_scale;
  int decoupled;  // 1 = AdamW, 0 = Adam (L2 added to the gradient)
};

__device__ __forceinline__ void adam_update(float& p, float& m, float& v, float g, const AdamArgs& a) {
  float gj = g * a.grad_scale;
  if (!a.decoupled) gj += a.wd * p;
  m = a.beta1 * m + (1.f - a.beta1) * gj;
  v = a.beta2 * v + (1.f - a.beta2) * gj * gj;
  const float mh = m / a.bc1, vh = v / a.bc2;
  float pj = p;
  if (a.decoupled) pj *= (1.f - a.lr * a.wd);
  p = pj - a.lr * mh / (sqrtf(vh) + a.eps);
}

// grad is bf16 or fp32; p/m/v fp32; optional bf16 copy of the updated weights. `skip` (device int)
// non-zero turns the launch into a no-op (loss-scaler found inf/nan).
template <typename G>
__global__ void adam_flat_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                                 const G* __restrict__ g, __nv_bfloat16* __restrict__ p_lp, long long n, AdamArgs a,
                                 const int* __restrict__ skip, const int* __restrict__ step_dev) {
  if (skip && *skip) return;
  if (step_dev) {   // step number kept on the device (a launch recorded in a CUDA graph is replayed with frozen arguments)
    const float t = (float)*step_dev;
    a.bc1 = 1.f - powf(a.beta1, t);
    a.bc2 = 1.f - powf(a.beta2, t);
  }
  const long long nvec = n >> 2;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec;
       i += (long long)gridDim.x * blockDim.x) {
    float4 pv = reinterpret_cast<float4*>(p)[i];
    float4 mv = reinterpret_cast<float4*>(m)[i];
    float4 vv = reinterpret_cast<float4*>(v)[i];
    float gr[4];
    if (sizeof(G) == 4) {
      float4 gv = reinterpret_cast<const float4*>(g)[i];
      gr[0] = gv.x; gr[1] = gv.y; gr[2] = gv.z; gr[3] = gv.w;
    } else {
      uint2 gu = reinterpret_cast<const uint2*>(g)[i];
      float2 a0 = unpack_bf16x2(gu.x), a1 = unpack_bf16x2(gu.y);
      gr[0] = a0.x; gr[1] = a0.y; gr[2] = a1.x; gr[3] = a1.y;
    }
    float* pp = reinterpret_cast<float*>(&pv);
    float* mp = reinterpret_cast<float*>(&mv);
    float* vp = reinterpret_cast<float*>(&vv);
#pragma unroll
    for (int j = 0; j < 4; ++j) adam_update(pp[j], mp[j], vp[j], gr[j], a);
    reinterpret_cast<float4*>(p)[i] = pv;
    reinterpret_cast<float4*>(m)[i] = mv;
    reinterpret_cast<float4*>(v)[i] = vv;
    if (p_lp) {
      uint2 o;
      o.x = pack_bf16x2(pp[0], pp[1]);
      o.y = pack_bf16x2(pp[2], pp[3]);
      reinterpret_cast<uint2*>(p_lp)[i] = o;
    }
  }
  // tail (n % 4) handled by the first threads of block 0
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const long long i = (nvec << 2) + threadIdx.x;
    const float gi = sizeof(G) == 4 ? reinterpret_cast<const float*>(g)[i]
                                    : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g)[i]);
    adam_update(p[i], m[i], v[i], gi, a);
    if (p_lp) p_lp[i] = __float2bfloat16(p[i]);
  }
}

// Adam / AdamW over many parameter tensors in one launch: master weights and moments are one flat buffer, every
// gradient and every bf16 weight is read and written where it lies. Bound by memory: 24 bytes per weight for master
// and moments plus the gradient and the bf16 copy, each moved once. Gathering the gradients into a flat fp32 buffer
// first and copying the weights out afterwards moved 40 bytes per bf16 weight instead of 28, in two launches per tensor:
// 50.4 M weights in 48 tensors took 879 us, this kernel takes 235 us (6.0 TB/s).
// The tensor table travels in the kernel's parameters (gradients move from step to step, and nothing has to be copied
// to the device or outlive the launch); a CTA finds its tensor by bisection over the first-CTA column.
constexpr int ADAM_MULTI_TENSORS = 100;                      // 100 table rows + arguments < 4 KB of parameters
constexpr int ADAM_MULTI_THREADS = 256, ADAM_MULTI_VECS = 2; // vectors of four in flight per thread and round
constexpr int ADAM_MULTI_CHUNK = ADAM_MULTI_THREADS * 4 * ADAM_MULTI_VECS * 2;

struct AdamTable {
  const void* grad[ADAM_MULTI_TENSORS];
  __nv_bfloat16* lp[ADAM_MULTI_TENSORS];       // bf16 weights to write, or null
  long long off[ADAM_MULTI_TENSORS];           // first element in the flat buffers, a multiple of four
  long long n[ADAM_MULTI_TENSORS];
  int first_cta[ADAM_MULTI_TENSORS];
  unsigned char grad_bf16[ADAM_MULTI_TENSORS];
  int count;
};

__global__ void __launch_bounds__(ADAM_MULTI_THREADS)
adam_multi_kernel(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v, const __grid_constant__ AdamTable tab,
                  const AdamArgs a) {
  int lo = 0, hi = tab.count;                  // last row whose first CTA is not behind this one
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tab.first_cta[mid] <= (int)blockIdx.x) lo = mid; else hi = mid;
  }
  const long long n = tab.n[lo], off = tab.off[lo];
  const long long e0 = (long long)((int)blockIdx.x - tab.first_cta[lo]) * ADAM_MULTI_CHUNK;
  const bool gb = tab.grad_bf16[lo] != 0;
  const void* grad = tab.grad[lo];
  __nv_bfloat16* lp = tab.lp[lo];
  // whole vectors only where gradient and bf16 weights start on a vector boundary (views may not)
  const bool wide = ((reinterpret_cast<uintptr_t>(grad) & (gb ? 7 : 15)) | (reinterpret_cast<uintptr_t>(lp) & 7)) == 0;
  p += off; m += off; v += off;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    float4 pv[ADAM_MULTI_VECS], mv[ADAM_MULTI_VECS], vv[ADAM_MULTI_VECS], gv[ADAM_MULTI_VECS];
    const long long e = e0 + ((long long)r * ADAM_MULTI_VECS * ADAM_MULTI_THREADS + threadIdx.x) * 4;
    bool full[ADAM_MULTI_VECS];
#pragma unroll
    for (int k = 0; k < ADAM_MULTI_VECS; ++k) {
      const long long i = e + (long long)k * ADAM_MULTI_THREADS * 4;
      full[k] = wide && i + 4 <= n;
      if (full[k]) {
        pv[k] = *reinterpret_cast<const float4*>(p + i);
        mv[k] = *reinterpret_cast<const float4*>(m + i);
        vv[k] = *reinterpret_cast<const float4*>(v + i);
        if (gb) {
          const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(grad) + i);
          const float2 x = unpack_bf16x2(u.x), y = unpack_bf16x2(u.y);
          gv[k] = make_float4(x.x, x.y, y.x, y.y);
        } else {
          gv[k] = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(grad) + i);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < ADAM_MULTI_VECS; ++k) {
      const long long i = e + (long long)k * ADAM_MULTI_THREADS * 4;
      if (full[k]) {
        adam_update(pv[k].x, mv[k].x, vv[k].x, gv[k].x, a);
        adam_update(pv[k].y, mv[k].y, vv[k].y, gv[k].y, a);
        adam_update(pv[k].z, mv[k].z, vv[k].z, gv[k].z, a);
        adam_update(pv[k].w, mv[k].w, vv[k].w, gv[k].w, a);
        *reinterpret_cast<float4*>(p + i) = pv[k];
        *reinterpret_cast<float4*>(m + i) = mv[k];
        *reinterpret_cast<float4*>(v + i) = vv[k];
        if (lp) *reinterpret_cast<uint2*>(lp + i) = make_uint2(pack_bf16x2(pv[k].x, pv[k].y), pack_bf16x2(pv[k].z, pv[k].w));
      } else {
        for (long long j = i; j < i + 4 && j < n; ++j) {
          const float gj = gb ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(grad)[j])
                              : reinterpret_cast<const float*>(grad)[j];
          adam_update(p[j], m[j], v[j], gj, a);
          if (lp) lp[j] = __float2bfloat16(p[j]);
        }
      }
    }
  }
}

template <typename G>
__global__ void sgd_flat_kernel(float* __restrict__ p, float* __restrict__ buf, const G* __restrict__ g,
                                __nv_bfloat16* __restrict__ p_lp, long long n, float lr, float momentum,
                                float dampening, float wd, int nesterov, int first_step, float grad_scale) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    float gj = (sizeof(G) == 4 ? reinterpret_cast<const float*>(g)[i]
                               : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g)[i])) *
               grad_scale;
    gj += wd * p[i];
    if (momentum != 0.f) {
      float b = first_step ? gj : momentum * buf[i] + (1.f - dampening) * gj;
      buf[i] = b;
      gj = nesterov ? gj + momentum * b : b;
    }
    const float pj = p[i] - lr * gj;
    p[i] = pj;
    if (p_lp) p_lp[i] = __float2bfloat16(pj);
  }
}

// Sum of squares of a flat gradient into out[0] (atomic), plus a non-finite flag into out[1].
template <typename G>
__global__ void sumsq_kernel(const G* __restrict__ g, long long n, float* __restrict__ out) {
  __shared__ float red[32];
  float acc = 0.f;
  int bad = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = sizeof(G) == 4 ? reinterpret_cast<const float*>(g)[i]
                                   : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(g)[i]);
    acc += v * v;
    bad |= !isfinite(v);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  bad = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = acc;
    if (bad) out[1] = 1.f;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (blockDim.x >> 5); ++w) t += red[w];
    atomicAdd(out, t);
  }
}

static inline int flat_grid(long long n) {
  long long g = (n + 1023) / 1024;
  // four CTAs (1024 threads) per SM at most: these kernels are HBM-bound and usually run beside compute kernels of another
  // stream, which must still find free thread slots and registers on every SM
  const long long cap = (long long)sm_count() * 4;
  return (int)(g < cap ? (g > 0 ? g : 1) : cap);
}

}  // namespace gf

using namespace gf;

// dlogits may equal logits (in place) or be null (loss only). ld = row pitch in elements. status: device int that receives a
// code when the bounded wait for a row runs out (that CTA's remaining rows are then not written).
GF_API int gf_xent_fused(const void* logits, const long long* targets, float* loss_rows, void* dlogits, int T, int V,
                         long long ld, float grad_scale, long long ignore_index, int* status, void* stream) {
  gf::enter();
  const long long v8 = ((long long)V + 7) / 8 * 8;
  if (V <= 0 || ld % 8 || ld < v8 || T <= 0 || !status) return GFH_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(logits) & 15) || (reinterpret_cast<uintptr_t>(dlogits) & 15)) return GFH_BAD_ARG;
  const size_t smem = (size_t)v8 * 2;
  if (smem > 200 * 1024) return GFH_TOO_LARGE;
  static gf::DeviceMax configured;
  if (smem > configured.get()) {
    if (cudaFuncSetAttribute(xent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return GFH_CUDA;
    configured.set(smem);
  }
  long long per_sm = (long long)(XENT_SMEM / (smem + 2048));   // 1 KB of static and reserved shared memory each, rounded up
  per_sm = per_sm < 1 ? 1 : per_sm > XENT_CTAS ? XENT_CTAS : per_sm;
  const long long most = per_sm * sm_count();
  xent_kernel<<<(unsigned)(T < most ? T : most), XENT_THREADS, smem, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)logits, targets, loss_rows, (__nv_bfloat16*)dlogits, T, V, ld, grad_scale, ignore_index, status);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// grad_dtype: 0 fp32, 1 bf16. p_lp may be null. skip may be null.
// step_dev (may be null): device int holding the step number; when given, `step` is ignored.
GF_API int gf_adam_flat_dev(float* p, float* m, float* v, const void* g, void* p_lp, long long n, float lr, float beta1,
                            float beta2, float eps, float wd, int step, float grad_scale, int decoupled,
                            int grad_dtype, const int* skip, const int* step_dev, void* stream) {
  gf::enter();
  if (n <= 0) return GFH_OK;
  static gf::DeviceOnce configured;
  if (configured.todo()) {
    prefer_max_smem(adam_flat_kernel<__nv_bfloat16>);
    prefer_max_smem(adam_flat_kernel<float>);
    configured.mark();
  }
  AdamArgs a;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.wd = wd; a.grad_scale = grad_scale;
  a.bc1 = 1.f - powf(beta1, (float)step);
  a.bc2 = 1.f - powf(beta2, (float)step);
  a.decoupled = decoupled;
  if (grad_dtype == 1)
    adam_flat_kernel<__nv_bfloat16><<<flat_grid(n), 256, 0, (cudaStream_t)stream>>>(
        p, m, v, (const __nv_bfloat16*)g, (__nv_bfloat16*)p_lp, n, a, skip, step_dev);
  else
    adam_flat_kernel<float><<<flat_grid(n), 256, 0, (cudaStream_t)stream>>>(
        p, m, v, (const float*)g, (__nv_bfloat16*)p_lp, n, a, skip, step_dev);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// Whether a launch over this table would write memory that it also reads or writes elsewhere: weights over one storage (the
// caller's copy back has an order, the launch has none), a gradient over a weight or over the flat buffers. Host only.
static bool adam_table_overlaps(const float* p, const float* m, const float* v, const long long* table, int count) {
  struct Span {
    unsigned long long lo, hi;
    bool written;
  };
  Span* s = new (std::nothrow) Span[2 * (size_t)count + 3];
  if (!s) return true;
  size_t k = 0;
  long long all = 0;
  for (int i = 0; i < count; ++i) {
    const long long *r = table + 5 * i, n = r[3];
    if (n <= 0) continue;
    if (r[0]) all = all < r[2] + n ? r[2] + n : all;
    if (r[1]) s[k++] = {(unsigned long long)r[1], (unsigned long long)(r[1] + n * (r[0] ? 2 : r[4])), true};
    if (r[0]) s[k++] = {(unsigned long long)r[0], (unsigned long long)(r[0] + n * (r[4] ? 2 : 4)), false};
  }
  for (const float* f : {p, m, v})
    if (all) s[k++] = {(unsigned long long)f, (unsigned long long)(f + all), true};
  std::sort(s, s + k, [](const Span& a, const Span& b) { return a.lo < b.lo; });
  unsigned long long end = 0, end_written = 0;
  bool hit = false;
  for (size_t i = 0; i < k && !hit; ++i) {
    hit = s[i].lo < (s[i].written ? end : end_written);
    if (s[i].hi > end) end = s[i].hi;
    if (s[i].written && s[i].hi > end_written) end_written = s[i].hi;
  }
  delete[] s;
  return hit;
}
GF_API int gf_adam_table_overlaps(const float* p, const float* m, const float* v, const long long* table, int count) {
  return count > 0 && table && adam_table_overlaps(p, m, v, table, count) ? 1 : 0;
}

// Adam / AdamW over `count` tensors. p / m / v: fp32 flat buffers; table (host memory, read before the call returns):
// five values per tensor {gradient pointer, bf16 weight pointer or 0, first element in the flat buffers (a multiple of
// four), number of elements, 1 when the gradient is bf16 and 0 when it is fp32}. A row without a gradient stands for a weight
// that the caller writes itself, fifth value its bytes per element. GFH_OVERLAP, and nothing launched, when adam_table_overlaps.
GF_API int gf_adam_multi(float* p, float* m, float* v, const long long* table, int count, float lr, float beta1,
                         float beta2, float eps, float wd, int step, float grad_scale, int decoupled, void* stream) {
  gf::enter();
  if (count < 0 || (count && !table)) return GFH_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15)
    return GFH_BAD_ARG;
  AdamArgs a;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.wd = wd; a.grad_scale = grad_scale;
  a.bc1 = 1.f - powf(beta1, (float)step);
  a.bc2 = 1.f - powf(beta2, (float)step);
  a.decoupled = decoupled;
  for (int i = 0; i < count; ++i)
    if (table[5 * i + 2] < 0 || (table[5 * i + 2] & 3) || table[5 * i + 3] < 0) return GFH_BAD_ARG;
  if (count && adam_table_overlaps(p, m, v, table, count)) return GFH_OVERLAP;
  AdamTable t;
  t.count = 0;
  long long ctas = 0;
  int launches = 0;
  for (int i = 0; i <= count; ++i) {
    const long long n = i < count && table[5 * i] ? table[5 * i + 3] : 0;
    const long long need = (n + ADAM_MULTI_CHUNK - 1) / ADAM_MULTI_CHUNK;
    if (need > 0x7fffffffLL) return GFH_TOO_LARGE;
    if (t.count && (i == count || t.count == ADAM_MULTI_TENSORS || ctas + need > 0x7fffffffLL)) {
      adam_multi_kernel<<<(unsigned)ctas, ADAM_MULTI_THREADS, 0, (cudaStream_t)stream>>>(p, m, v, t, a);
      ++launches;
      t.count = 0;
      ctas = 0;
    }
    if (i == count || n == 0) continue;
    const int k = t.count++;
    t.grad[k] = reinterpret_cast<const void*>(table[5 * i]);
    t.lp[k] = reinterpret_cast<__nv_bfloat16*>(table[5 * i + 1]);
    t.off[k] = table[5 * i + 2];
    t.n[k] = n;
    t.first_cta[k] = (int)ctas;
    t.grad_bf16[k] = table[5 * i + 4] != 0;
    ctas += need;
  }
  if (launches > 1) gf::note_extra_launches(launches - 1);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

GF_API int gf_adam_flat(float* p, float* m, float* v, const void* g, void* p_lp, long long n, float lr, float beta1,
                        float beta2, float eps, float wd, int step, float grad_scale, int decoupled, int grad_dtype,
                        const int* skip, void* stream) {
  return gf_adam_flat_dev(p, m, v, g, p_lp, n, lr, beta1, beta2, eps, wd, step, grad_scale, decoupled, grad_dtype,
                          skip, nullptr, stream);
}

GF_API int gf_sgd_flat(float* p, float* buf, const void* g, void* p_lp, long long n, float lr, float momentum,
                       float dampening, float wd, int nesterov, int first_step, float grad_scale, int grad_dtype,
                       void* stream) {
  gf::enter();
  if (n <= 0) return GFH_OK;
  if (grad_dtype == 1)
    sgd_flat_kernel<__nv_bfloat16><<<flat_grid(n), 256, 0, (cudaStream_t)stream>>>(
        p, buf, (const __nv_bfloat16*)g, (__nv_bfloat16*)p_lp, n, lr, momentum, dampening, wd, nesterov, first_step,
        grad_scale);
  else
    sgd_flat_kernel<float><<<flat_grid(n), 256, 0, (cudaStream_t)stream>>>(
        p, buf, (const float*)g, (__nv_bfloat16*)p_lp, n, lr, momentum, dampening, wd, nesterov, first_step,
        grad_scale);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}

// out: fp32[2] = {sum of squares (accumulated), non-finite flag}; caller zeroes it first.
GF_API int gf_grad_sumsq(const void* g, long long n, float* out, int grad_dtype, void* stream) {
  gf::enter();
  if (n <= 0) return GFH_OK;
  if (grad_dtype == 1)
    sumsq_kernel<__nv_bfloat16><<<flat_grid(n), 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)g, n, out);
  else
    sumsq_kernel<float><<<flat_grid(n), 256, 0, (cudaStream_t)stream>>>((const float*)g, n, out);
  return cudaGetLastError() == cudaSuccess ? GFH_OK : GFH_CUDA;
}
