// Host interface of the GEMM (gemm.cu) for other translation units of this library.
#pragma once
#include "common.cuh"

namespace ttcd {

// C[b] = alpha * rowscale * A[b] B[b]^T (+ beta * Cin[b]), bf16 operands, as the file comment of gemm.cu says.
struct GemmCall {
  const void* a = nullptr; const void* b = nullptr; void* c = nullptr;
  const void* c_in = nullptr; const void* row_scale = nullptr;
  int64_t M = 0, N = 0, K = 0, batch = 1, lda = 0, ldb = 0, ldc = 0, stride_a = 0, stride_b = 0, stride_c = 0;
  int a_mn = 0, b_mn = 0, out_fp32 = 0;
  float alpha = 1.f, beta = 0.f;
  float* lse_part = nullptr;
  // The rows of B may come from up to three matrices of their own (K-major, batch 1): rows [0, n1) from b, [n1, n1 + n2) from b2, the
  // rest from b3; n1 = 0: all from b.  n1 and n2 have to be multiples of a tile's width (64 at least).
  const void* b2 = nullptr; const void* b3 = nullptr;
  int64_t n1 = 0, n2 = 0;
  // bf16 output, c_in with beta 1: the product is rounded before c_in is added (the sum is rounded again)
  int round_first = 0;
  // b: gate, b2: up, [N, K] each, K-major, batch 1: C = silu(A b^T) * (A b2^T), both products rounded to bf16 first
  int swiglu = 0;
};
int gemm_run(const GemmCall& call, cudaStream_t stream);
// Whether B's rows from matrices of n1, n2 and n3 rows make the product of M rows slower than putting them side by side first does.
bool gemm_pieces_slow(int64_t M, int64_t K, int64_t n1, int64_t n2, int64_t n3);

}  // namespace ttcd
