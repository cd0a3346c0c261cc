// Launcher of the few-row GEMM (gemm_rows.cu) for the other launchers of the library.
#pragma once
#include <cuda_runtime.h>

namespace gf {

enum RowsInput : int {
  ROWS_PLAIN = 0,     // X [M, K]
  ROWS_RMSNORM = 1,   // RMS norm of X [M, K] with weight `norm_w` and `eps`
  ROWS_SWIGLU = 2,    // silu(X[:, :K]) * X[:, K:] of X [M, 2 K]; a kernel in front of a plain product is faster (see gemm_rows.cu)
};

struct RowsGemm {
  const void* X;
  long long ldx;
  const void* W;          // [N, K], pitch ldw
  long long ldw;
  void* C;
  long long ldc;
  int out_fp32, M, N, K;
  RowsInput input;
  const void* norm_w;
  float eps;
  const void* bias;
  const void* residual;
  long long ldr;
  float alpha;
  int relu;
  int* status;
};

constexpr int ROWS_MAX_M = 64;
constexpr int ROWS_MAX_M_FUSED = 16;     // with an input other than ROWS_PLAIN

// Whether the kernel takes the operands: at most 64 rows, both K-major, whole 16-byte vectors.
bool gemm_rows_takes(const void* X, long long ldx, const void* W, long long ldw, int M, int N, int K);
// `chained`: the launch in front of this one on `stream` is a kernel of the same call that has not written W and whose own
// predecessors were complete when it started (see griddepcontrol in gemm_rows.cu). 0 otherwise.
int gemm_rows_run(const RowsGemm& g, int chained, cudaStream_t stream);

}  // namespace gf
