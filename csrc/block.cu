// A plain pre-norm decoder block over a prompt (inference) from one call: the launches of RMSNorm, the fused q|k|v projection,
// per-head norm and rotary, attention, o_proj + residual, RMSNorm, gate|up + SwiGLU, down_proj + residual, issued from C++.  A
// block took ~370 us of Python between eleven launches, so that a chat-sized prompt (300 tokens, 28 blocks) spent 10.4 ms on
// 2.7 ms of device work.  The roundings are those of the block run module by module (custom_models/ipttcd/
// modeling_ipttcdv9.py:794-850 for the order of the parts).
#include "gemm.cuh"

extern "C" {
int ttcd_rmsnorm_fwd(const void* x, const void* res, const void* w, void* y, void* sum_out, float* rstd, long long rows, int D,
                     float eps, void* stream_ptr);
int ttcd_qk_norm_rope_fwd(const void* q_in, long long ldq, const void* k_in, long long ldk, void* q_out, long long ldqo, void* k_out,
                          long long ldko, const void* qw, const void* kw, const void* cos, const void* sin, const int* positions,
                          long long rows, int T, int pos_offset, int H, int HK, int D, int half, float eps, void* stream_ptr);
int ttcd_attn_fwd(const void* q, const void* k, const void* v, void* o_t, void* o_s, float* lse_t, float* lse_s, int B, int Tq, int Tk,
                  int H, int HK, int D, long long ldq, long long ldk, long long ldv, long long sq, long long sk, long long sv,
                  int window_t, int window_s, float scale, const int* seg_start, int form, void* stream_ptr);
}

// p: x, x_out, normed, rstd, qkv, q, k, o, lse, sum, z (device addresses; see below), the weights attn_norm, mlp_norm, Wq, Wk, Wv, Wo, Wg,
// Wu, Wd, q_norm, k_norm (or 0), cos, sin (or 0), then B, T, hidden, inter, H, HK, D, window (0: none), heads' rotary half, wide.
//   x, x_out, normed, sum [B T, hidden]; rstd [B T] fp32; qkv [B T, (H + 2 HK) D]; q [B T, H D]; k [B T, HK D]; o [B T, H D]; lse [B, H, T]
//   fp32; z [B T, inter]; normed may be x_out, sum may lie over q, and z over q and o.  k (after norm and rotary; untouched where there is neither) and
//   the last HK D columns of qkv are what a cache keeps.  wide [(H + 2 HK) D, hidden] (or 0): room for Wq, Wk and Wv side by side where
//   that is the faster way.  All bf16 contiguous and 16-byte aligned; B T >= 128, T >= 128, hidden and inter >= 128 and multiples of 8, D 64 or 128.
// f: eps of attn_norm, of mlp_norm, of q_norm / k_norm, the scores' scale.
TTCD_EXPORT int ttcd_block_prefill(const long long* p, const float* f, void* stream_ptr) {
  using namespace ttcd;
  auto at = [&](int i) { return reinterpret_cast<void*>(p[i]); };
  const int64_t B = p[24], T = p[25], hidden = p[26], inter = p[27], H = p[28], HK = p[29], D = p[30];
  const int window = static_cast<int>(p[31]), half = static_cast<int>(p[32]);
  if (B < 1 || T < 128 || hidden < 128 || inter < 128 || hidden % 8 != 0 || inter % 8 != 0 || H < 1 || HK < 1 || H % HK != 0 ||
      (D != 64 && D != 128))
    return TTCD_ERR_ARG;
  for (int i = 0; i < 24; ++i)
    if ((p[i] == 0 && i < 20) || p[i] % 16 != 0) return TTCD_ERR_ARG;
  if (p[33] % 16 != 0) return TTCD_ERR_ARG;
  const int64_t rows = B * T, q_cols = H * D, kv_cols = HK * D, cols = q_cols + 2 * kv_cols;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  bf16* const qkv = static_cast<bf16*>(at(4));

  int rc = ttcd_rmsnorm_fwd(at(0), nullptr, at(11), at(2), nullptr, static_cast<float*>(at(3)), rows, static_cast<int>(hidden), f[0], stream);
  if (rc != TTCD_OK) return rc;
  GemmCall g;
  g.a = at(2); g.b = at(13); g.c = qkv; g.M = rows; g.N = cols; g.K = hidden; g.lda = g.ldb = hidden; g.ldc = cols; g.stride_c = rows * cols;
  if (p[14] != p[13] + q_cols * hidden * 2 || p[15] != p[14] + kv_cols * hidden * 2) {     // three matrices, not one
    if (p[33] != 0 && gemm_pieces_slow(rows, hidden, q_cols, kv_cols, kv_cols)) {
      int64_t row = 0;
      for (int i = 0; i < 3; ++i) {
        const int64_t n = i == 0 ? q_cols : kv_cols;
        TTCD_CUDA_CHECK(cudaMemcpyAsync(static_cast<bf16*>(at(33)) + row * hidden, at(13 + i), n * hidden * 2, cudaMemcpyDeviceToDevice, stream));
        row += n;
      }
      g.b = at(33);
    } else {
      g.b2 = at(14); g.b3 = at(15); g.n1 = q_cols; g.n2 = kv_cols;
    }
  }
  rc = gemm_run(g, stream);
  if (rc != TTCD_OK) return rc;
  const bf16 *q = qkv, *k = qkv + q_cols;
  int64_t ldq = cols, ldk = cols;
  if (p[20] != 0 || p[22] != 0) {
    rc = ttcd_qk_norm_rope_fwd(qkv, cols, qkv + q_cols, cols, at(5), q_cols, at(6), kv_cols, at(20), at(21), at(22), at(23), nullptr, rows,
                               static_cast<int>(T), 0, static_cast<int>(H), static_cast<int>(HK), static_cast<int>(D), half, f[2], stream);
    if (rc != TTCD_OK) return rc;
    q = static_cast<bf16*>(at(5)); k = static_cast<bf16*>(at(6));
    ldq = q_cols; ldk = kv_cols;
  }
  rc = ttcd_attn_fwd(q, k, qkv + q_cols + kv_cols, at(7), nullptr, static_cast<float*>(at(8)), nullptr, static_cast<int>(B),
                     static_cast<int>(T), static_cast<int>(T), static_cast<int>(H), static_cast<int>(HK), static_cast<int>(D), ldq, ldk, cols,
                     T * ldq, T * ldk, T * cols, window, window, f[3], nullptr, 0, stream);
  if (rc != TTCD_OK) return rc;
  GemmCall o;
  o.a = at(7); o.b = at(16); o.c = at(9); o.c_in = at(0); o.beta = 1.f; o.round_first = 1;
  o.M = rows; o.N = hidden; o.K = q_cols; o.lda = o.ldb = q_cols; o.ldc = hidden; o.stride_c = rows * hidden;
  rc = gemm_run(o, stream);
  if (rc != TTCD_OK) return rc;
  rc = ttcd_rmsnorm_fwd(at(9), nullptr, at(12), at(2), nullptr, static_cast<float*>(at(3)), rows, static_cast<int>(hidden), f[1], stream);
  if (rc != TTCD_OK) return rc;
  GemmCall u;
  u.a = at(2); u.b = at(17); u.b2 = at(18); u.c = at(10); u.swiglu = 1;
  u.M = rows; u.N = inter; u.K = hidden; u.lda = u.ldb = hidden; u.ldc = inter; u.stride_c = rows * inter;
  rc = gemm_run(u, stream);
  if (rc != TTCD_OK) return rc;
  GemmCall d;
  d.a = at(10); d.b = at(19); d.c = at(1); d.c_in = at(9); d.beta = 1.f; d.round_first = 1;
  d.M = rows; d.N = hidden; d.K = inter; d.lda = d.ldb = inter; d.ldc = hidden; d.stride_c = rows * hidden;
  return gemm_run(d, stream);
}
