// Row-wise cross-entropy with in-place gradient, LSE merge of two partial attention results, fused
// AdamW over flat shards (with device-side clip coefficient and skip flag, so no host sync) and the
// squared-norm reduction used for gradient clipping.  Replaces
// fla/modules/fused_linear_cross_entropy.py:33-190, profiling/lse_dual_attn.py:106-160 and
// torch._fused_adamw_ / clip_grad_norm_ on the reference's training path.
#include "common.cuh"

#include <algorithm>

namespace ttcd {

__device__ __forceinline__ float block_reduce(float v, float* scratch, bool is_max) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  v = is_max ? warp_max(v) : warp_sum(v);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float t = lane < warps ? scratch[lane] : (is_max ? -INFINITY : 0.f);
    t = is_max ? warp_max(t) : warp_sum(t);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  const float out = scratch[32];
  __syncthreads();
  return out;
}

// One block per row of logits [rows][ld] (bf16).  With eps = label smoothing and zeta = the weight of lse^2:
//   loss_row[row] = lse - (1 - eps) logit[label] - eps mean(logits) + zeta lse^2      (0 when the label is ignored)
// and, when write_grad, the row is overwritten with its gradient times (*grad_scale):
//   softmax (1 + 2 zeta lse) - (1 - eps) onehot - eps / V
// l2_factor > 0 adds the l2-warp term on EVERY row (ignored ones too, as the reference's fused linear-CE does,
// fla/modules/fused_linear_cross_entropy.py:250-283): max logit * l2_factor * (*grad_scale) at the arg-max column
// (the lowest column on ties); the loss value is unchanged by it.
// A block of 256 threads does the work of one of 1024: a thread has CE_U accumulators, so that its CE_U loads are in flight
// together and several rows share an SM (one's reductions hide behind another's loads) while every sum keeps its order; the
// outputs of the two are the same bit by bit.  With fewer rows than SMs there is nothing to share, and a long row takes what
// one block's threads can have in flight: those get 1024.  us, 1024 | 256 threads: 16384 x 32000: 704 | 615, with lse_part
// 513 | 426; 9472 x 151936: 1711 | 1570, 1084 | 981;  128 x 32000: 8.3 | 9.8, 150 x 32000: 13.4 | 13.0;  128 x 151936:
// 26.5 | 37.0, 300 x 151936: 73 | 80, 450 x 151936: 102 | 103;  128 x 4096: 3.9 | 4.0, 150 x 4096: 5.1 | 4.5.
// The gradient goes to `grad` (rows ld apart like the logits; it may be `logits` itself).
constexpr int CE_ROW = 1024;

// One value per thread of a CE_ROW-thread block, v[u] for thread u * THREADS + threadIdx.x; block_reduce's order.
template <int THREADS>
__device__ __forceinline__ float ce_reduce(float (&v)[CE_ROW / THREADS], float* scratch, bool is_max) {
  constexpr int CE_U = CE_ROW / THREADS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int u = 0; u < CE_U; ++u) {
    const float w = is_max ? warp_max(v[u]) : warp_sum(v[u]);
    if (lane == 0) scratch[u * (THREADS / 32) + warp] = w;
  }
  __syncthreads();
  if (warp == 0) {
    static_assert(CE_ROW == 1024, "one value per lane below");
    const float t = is_max ? warp_max(scratch[lane]) : warp_sum(scratch[lane]);
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  const float out = scratch[32];
  __syncthreads();
  return out;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) ce_rows_kernel(const bf16* logits, bf16* grad, const int64_t* __restrict__ labels,
                                                       float* __restrict__ loss_row, float* __restrict__ lse_row,
                                                       const float* __restrict__ grad_scale, int V, int64_t ld,
                                                       int ignore_index, int write_grad, float eps, float zeta,
                                                       float l2_factor, const float2* __restrict__ lse_part, int n_parts) {
  constexpr int CE_U = CE_ROW / THREADS;
  __shared__ float scratch[33];
  const int64_t row = blockIdx.x;
  const bf16* lr = logits + row * ld;
  bf16* gr = grad + row * ld;
  const int64_t label = labels[row];
  const int nvec = V / 8;
  float m[CE_U], s[CE_U], sumx[CE_U];
  int arg[CE_U];
#pragma unroll
  for (int u = 0; u < CE_U; ++u) { m[u] = -INFINITY; s[u] = sumx[u] = 0.f; arg[u] = 0; }
  // the producing GEMM left (max, sum) per column tile of this row: merge them instead of reading the row
  const bool have_parts = lse_part != nullptr;
  if (have_parts) {
    for (int base = threadIdx.x; base < n_parts; base += CE_ROW) {
#pragma unroll
      for (int u = 0; u < CE_U; ++u) {
        const int i = base + u * THREADS;
        if (i >= n_parts) break;
        const float2 t = lse_part[row * n_parts + i];
        if (t.x > m[u]) {
          s[u] *= __expf(m[u] - t.x);
          m[u] = t.x;
        }
        if (t.x != -INFINITY) s[u] += t.y * __expf(t.x - m[u]);
      }
    }
  } else {
    for (int base = threadIdx.x; base < nvec; base += CE_ROW) {
      uint4 raws[CE_U];
#pragma unroll
      for (int u = 0; u < CE_U; ++u) {
        const int i = base + u * THREADS;
        if (i < nvec) raws[u] = *reinterpret_cast<const uint4*>(lr + i * 8);
      }
#pragma unroll
      for (int u = 0; u < CE_U; ++u) {
        const int i = base + u * THREADS;
        if (i >= nvec) break;
        const uint32_t w[4] = {raws[u].x, raws[u].y, raws[u].z, raws[u].w};
        float f[8];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 t = unpack_bf16(w[k]);
          f[2 * k] = t.x;
          f[2 * k + 1] = t.y;
        }
        float lm = f[0];
        int la = 0;
#pragma unroll
        for (int k = 1; k < 8; ++k)
          if (f[k] > lm) { lm = f[k]; la = k; }
        if (lm > m[u]) {
          s[u] *= __expf(m[u] - lm);
          m[u] = lm;
          arg[u] = i * 8 + la;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          s[u] += __expf(f[k] - m[u]);
          sumx[u] += f[k];
        }
      }
    }
#pragma unroll
    for (int u = 0; u < CE_U; ++u) {
      const int i = nvec * 8 + threadIdx.x + u * THREADS;       // fewer than 8 columns are left
      if (i < V) {
        const float f = __bfloat162float(lr[i]);
        if (f > m[u]) {
          s[u] *= __expf(m[u] - f);
          m[u] = f;
          arg[u] = i;
        }
        s[u] += __expf(f - m[u]);
        sumx[u] += f;
      }
    }
  }
  const float gm = ce_reduce<THREADS>(m, scratch, true);
#pragma unroll
  for (int u = 0; u < CE_U; ++u) s[u] = (m[u] == -INFINITY) ? 0.f : s[u] * __expf(m[u] - gm);
  const float gs = ce_reduce<THREADS>(s, scratch, false);
  const float lse = gm + __logf(gs);
  float mean_x = 0.f;
  if (eps != 0.f) mean_x = ce_reduce<THREADS>(sumx, scratch, false) / static_cast<float>(V);
  int arg_col = -1;
  if (l2_factor != 0.f && write_grad) {       // column indices are below 2^24: exact as floats
#pragma unroll
    for (int u = 0; u < CE_U; ++u) m[u] = m[u] == gm ? -static_cast<float>(arg[u]) : -INFINITY;
    arg_col = -static_cast<int>(ce_reduce<THREADS>(m, scratch, true));
  }
  const bool valid = label != ignore_index && label >= 0 && label < V;
  if (threadIdx.x == 0) {
    loss_row[row] = valid ? lse - (1.f - eps) * __bfloat162float(lr[label]) - eps * mean_x + zeta * lse * lse : 0.f;
    if (lse_row != nullptr) lse_row[row] = lse;
  }
  if (!write_grad) return;
  const float gsc = *grad_scale;
  const float scale = valid ? gsc : 0.f;
  const float pw = 1.f + 2.f * zeta * lse, hot = 1.f - eps, flat = eps / static_cast<float>(V);
  const float warp_term = gm * l2_factor * gsc;
  __syncthreads();  // label logit read above before the row is overwritten
  for (int base = threadIdx.x; base < nvec; base += CE_ROW) {
    uint4 raws[CE_U];
#pragma unroll
    for (int u = 0; u < CE_U; ++u) {
      const int i = base + u * THREADS;
      if (i < nvec) raws[u] = *reinterpret_cast<const uint4*>(lr + i * 8);
    }
#pragma unroll
    for (int u = 0; u < CE_U; ++u) {
      const int i = base + u * THREADS;
      if (i >= nvec) break;
      uint32_t w[4] = {raws[u].x, raws[u].y, raws[u].z, raws[u].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float2 t = unpack_bf16(w[k]);
        const int c = i * 8 + 2 * k;
        t.x = (__expf(t.x - lse) * pw - (c == label ? hot : 0.f) - flat) * scale + (c == arg_col ? warp_term : 0.f);
        t.y = (__expf(t.y - lse) * pw - (c + 1 == label ? hot : 0.f) - flat) * scale + (c + 1 == arg_col ? warp_term : 0.f);
        w[k] = pack_bf16(t.x, t.y);
      }
      *reinterpret_cast<uint4*>(gr + i * 8) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  for (int i = nvec * 8 + threadIdx.x; i < V; i += blockDim.x) {
    const float f = __bfloat162float(lr[i]);
    gr[i] = __float2bfloat16((__expf(f - lse) * pw - (i == label ? hot : 0.f) - flat) * scale + (i == arg_col ? warp_term : 0.f));
  }
}

// out = merge of two partial softmax results over disjoint key sets.
// o_*: [rows][H][D] bf16, lse_*: [B][H][T] fp32 with rows = B*T; one warp per (row, head).
__global__ void __launch_bounds__(256) lse_merge_kernel(const bf16* __restrict__ oa, const float* __restrict__ la,
                                                        const bf16* __restrict__ ob, const float* __restrict__ lb,
                                                        bf16* __restrict__ out, float* __restrict__ lse_out,
                                                        int64_t B, int T, int H, int D) {
  const int lane = threadIdx.x & 31;
  const int64_t item = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= B * T * H) return;
  const int h = static_cast<int>(item % H);
  const int64_t bt = item / H;
  const int64_t b = bt / T, t = bt % T;
  const int64_t li = (b * H + h) * T + t;
  const float a = la[li], c = lb[li];
  float m = fmaxf(a, c);
  if (m == -INFINITY) m = 0.f;
  const float wa = __expf(a - m), wb = __expf(c - m);
  const float inv = 1.f / fmaxf(wa + wb, 1e-38f);
  if (lane == 0 && lse_out != nullptr) lse_out[li] = m + __logf(fmaxf(wa + wb, 1e-38f));
  const int64_t base = item * D;
  for (int d = lane * 2; d < D; d += 64) {
    const float2 x = unpack_bf16(*reinterpret_cast<const uint32_t*>(oa + base + d));
    const float2 y = unpack_bf16(*reinterpret_cast<const uint32_t*>(ob + base + d));
    *reinterpret_cast<uint32_t*>(out + base + d) =
        pack_bf16((x.x * wa + y.x * wb) * inv, (x.y * wa + y.y * wb) * inv);
  }
}

// Fused AdamW on a flat fp32 master shard.  grad is bf16 or fp32.  coef (device scalar, may be
// null) multiplies the gradient (clip); skip (device int, may be null) != 0 leaves everything as is.
// VEC: four elements per access (every array 16-byte aligned, bf16 ones 8); the last n % 4 elements one by one.  For 128 K
// elements or more: below, a quarter of the threads is too few.  us, one | four per access, bf16 gradient: 1000: 2.1 | 2.6,
// 100 K: 2.6 | 2.7, 200 K: 3.2 | 3.0, 600 K: 5.8 | 3.8, 65.5 M: 410 | 308 (284 us of bytes).
template <typename GradT, bool VEC>
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p, const GradT* __restrict__ g,
                                                    float* __restrict__ m, float* __restrict__ v,
                                                    bf16* __restrict__ p_bf16, int64_t n, float lr, float beta1,
                                                    float beta2, float eps, float wd, float bc1, float bc2_sqrt,
                                                    const float* __restrict__ coef, const int* __restrict__ skip) {
  if (skip != nullptr && *skip != 0) return;
  const float c = coef != nullptr ? *coef : 1.f;
  const float step_size = lr / bc1;
  auto update = [&](float gi, float& pi, float& mi, float& vi) {
    gi *= c;
    pi *= 1.f - lr * wd;
    mi = beta1 * mi + (1.f - beta1) * gi;
    vi = beta2 * vi + (1.f - beta2) * gi * gi;
    pi -= step_size * mi / (sqrtf(vi) / bc2_sqrt + eps);
  };
  const int64_t first = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x, stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  if constexpr (VEC) {
    for (int64_t i = first; i < n / 4; i += stride) {
      float gi[4];
      if constexpr (sizeof(GradT) == 2) {
        const uint2 raw = reinterpret_cast<const uint2*>(g)[i];
        const float2 lo = unpack_bf16(raw.x), hi = unpack_bf16(raw.y);
        gi[0] = lo.x; gi[1] = lo.y; gi[2] = hi.x; gi[3] = hi.y;
      } else {
        const float4 raw = reinterpret_cast<const float4*>(g)[i];
        gi[0] = raw.x; gi[1] = raw.y; gi[2] = raw.z; gi[3] = raw.w;
      }
      float4 pv = reinterpret_cast<const float4*>(p)[i], mv = reinterpret_cast<const float4*>(m)[i], vv = reinterpret_cast<const float4*>(v)[i];
      update(gi[0], pv.x, mv.x, vv.x);
      update(gi[1], pv.y, mv.y, vv.y);
      update(gi[2], pv.z, mv.z, vv.z);
      update(gi[3], pv.w, mv.w, vv.w);
      reinterpret_cast<float4*>(p)[i] = pv;
      reinterpret_cast<float4*>(m)[i] = mv;
      reinterpret_cast<float4*>(v)[i] = vv;
      if (p_bf16 != nullptr) reinterpret_cast<uint2*>(p_bf16)[i] = make_uint2(pack_bf16(pv.x, pv.y), pack_bf16(pv.z, pv.w));
    }
  }
  for (int64_t i = (VEC ? n / 4 * 4 : 0) + first; i < n; i += stride) {
    float gi;
    if constexpr (sizeof(GradT) == 2) gi = __bfloat162float(g[i]);
    else gi = g[i];
    float pi = p[i], mi = m[i], vi = v[i];
    update(gi, pi, mi, vi);
    p[i] = pi;
    m[i] = mi;
    v[i] = vi;
    if (p_bf16 != nullptr) p_bf16[i] = __float2bfloat16(pi);
  }
}

// Muon around the orthogonalisation, one launch per matrix on each side (a dozen element-wise launches before).
// Before it: g = grad * coef; m = momentum m + g, kept unless skip; out = bf16(nesterov ? g + momentum m : m).
// After it: p = p decay - rate u, kept unless skip; p_bf16 (may be null) = the weights after the step.
// The roundings are those of the separate operations (product and sum on their own, scaled addition fused).
struct MuonPreParams {
  const float* grad; float* mom; bf16* out; const float* coef; const int* skip;
  int64_t n; float momentum; int nesterov;
};
struct MuonPostParams {
  const bf16* u; float* p; bf16* p_bf16; const int* skip;
  int64_t n; float decay, rate;
};
template <int V>
__global__ void __launch_bounds__(256) muon_pre_kernel(const MuonPreParams a) {
  const float c = a.coef != nullptr ? *a.coef : 1.f;
  const bool keep = a.skip == nullptr || *a.skip == 0;
  for (int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * V; i < a.n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x * V) {
    float g[V], m[V];
    if constexpr (V == 4) {
      const float4 gv = *reinterpret_cast<const float4*>(a.grad + i), mv = *reinterpret_cast<const float4*>(a.mom + i);
      g[0] = gv.x; g[1] = gv.y; g[2] = gv.z; g[3] = gv.w;
      m[0] = mv.x; m[1] = mv.y; m[2] = mv.z; m[3] = mv.w;
    } else {
      g[0] = a.grad[i];
      m[0] = a.mom[i];
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      if (a.coef != nullptr) g[k] = __fmul_rn(g[k], c);
      m[k] = __fadd_rn(__fmul_rn(m[k], a.momentum), g[k]);
      g[k] = a.nesterov ? fmaf(a.momentum, m[k], g[k]) : m[k];
    }
    if constexpr (V == 4) {
      if (keep) *reinterpret_cast<float4*>(a.mom + i) = make_float4(m[0], m[1], m[2], m[3]);
      *reinterpret_cast<uint2*>(a.out + i) = make_uint2(pack_bf16(g[0], g[1]), pack_bf16(g[2], g[3]));
    } else {
      if (keep) a.mom[i] = m[0];
      a.out[i] = __float2bfloat16(g[0]);
    }
  }
}
template <int V>
__global__ void __launch_bounds__(256) muon_post_kernel(const MuonPostParams a) {
  const bool keep = a.skip == nullptr || *a.skip == 0;
  for (int64_t i = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * V; i < a.n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x * V) {
    float u[V], p[V];
    if constexpr (V == 4) {
      const uint2 uv = *reinterpret_cast<const uint2*>(a.u + i);
      const float2 lo = unpack_bf16(uv.x), hi = unpack_bf16(uv.y);
      const float4 pv = *reinterpret_cast<const float4*>(a.p + i);
      u[0] = lo.x; u[1] = lo.y; u[2] = hi.x; u[3] = hi.y;
      p[0] = pv.x; p[1] = pv.y; p[2] = pv.z; p[3] = pv.w;
    } else {
      u[0] = __bfloat162float(a.u[i]);
      p[0] = a.p[i];
    }
    if (keep) {
#pragma unroll
      for (int k = 0; k < V; ++k) p[k] = fmaf(-a.rate, u[k], __fmul_rn(p[k], a.decay));
    }
    if constexpr (V == 4) {
      if (keep) *reinterpret_cast<float4*>(a.p + i) = make_float4(p[0], p[1], p[2], p[3]);
      if (a.p_bf16 != nullptr) *reinterpret_cast<uint2*>(a.p_bf16 + i) = make_uint2(pack_bf16(p[0], p[1]), pack_bf16(p[2], p[3]));
    } else {
      if (keep) a.p[i] = p[0];
      if (a.p_bf16 != nullptr) a.p_bf16[i] = __float2bfloat16(p[0]);
    }
  }
}

// out[0] += sum(x^2) (atomicAdd of per-block partials; zero `out` beforehand).
template <typename T>
__global__ void __launch_bounds__(256) sumsq_kernel(const T* __restrict__ x, int64_t n, float* __restrict__ out) {
  __shared__ float scratch[33];
  float acc = 0.f;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float f;
    if constexpr (sizeof(T) == 2) f = __bfloat162float(x[i]);
    else f = x[i];
    acc += f * f;
  }
  acc = block_reduce(acc, scratch, false);
  if (threadIdx.x == 0) atomicAdd(out, acc);
}

// y[i] = x[i] * scale (+ y[i] when accumulate): bucket cast/scale used by the gradient path.
template <typename TI, typename TO>
__global__ void __launch_bounds__(256) cast_scale_kernel(const TI* __restrict__ x, TO* __restrict__ y, int64_t n,
                                                         float scale, int accumulate) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    float f;
    if constexpr (sizeof(TI) == 2) f = __bfloat162float(x[i]);
    else f = x[i];
    f *= scale;
    if constexpr (sizeof(TO) == 2) {
      if (accumulate) f += __bfloat162float(y[i]);
      y[i] = __float2bfloat16(f);
    } else {
      if (accumulate) f += y[i];
      y[i] = f;
    }
  }
}

// y = x * (*factor): a gradient times the scalar that arrives from downstream, 16 bytes per access (the broadcast
// multiplication of the library ran at 1.9 TB/s on the 2.1 GB of a 32768 x 32000 logits gradient).
__global__ void __launch_bounds__(256) scale_by_kernel(const bf16* __restrict__ x, bf16* __restrict__ y,
                                                       const float* __restrict__ factor, int64_t nvec) {
  const float f = *factor;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const uint4 raw = reinterpret_cast<const uint4*>(x)[i];
    const float2 a = unpack_bf16(raw.x), b = unpack_bf16(raw.y), c = unpack_bf16(raw.z), d = unpack_bf16(raw.w);
    reinterpret_cast<uint4*>(y)[i] = make_uint4(pack_bf16(a.x * f, a.y * f), pack_bf16(b.x * f, b.y * f),
                                                pack_bf16(c.x * f, c.y * f), pack_bf16(d.x * f, d.y * f));
  }
}

}  // namespace ttcd

using namespace ttcd;

static unsigned flat_grid(long long n) {
  return static_cast<unsigned>(std::max<long long>(1, std::min<long long>((n + 255) / 256, 148LL * 16)));
}

// logits: [rows][ld] bf16; labels: int64 [rows]; grad (used when write_grad): [rows][ld] bf16, may be logits.
// lse_part (may be null): fp32 [rows][n_parts][2] left by ttcd_gemm_bf16_lse for these logits; the first pass over the
// row is then skipped (not with label smoothing or the l2-warp term, which need the row's mean / arg-max).
TTCD_EXPORT int ttcd_ce_rows(const void* logits, void* grad, const long long* labels, float* loss_row, float* lse_row,
                             const float* grad_scale, long long rows, int V, long long ld, int ignore_index,
                             int write_grad, float label_smoothing, float lse_square_scale, float l2_factor,
                             const float* lse_part, int n_parts, void* stream_ptr) {
  if (rows <= 0 || V <= 0 || ld % 8 != 0 || (write_grad && (grad_scale == nullptr || grad == nullptr))) return TTCD_ERR_ARG;
  if (label_smoothing < 0.f || label_smoothing >= 1.f || V >= (1 << 24)) return TTCD_ERR_ARG;
  if (lse_part != nullptr && (n_parts <= 0 || label_smoothing != 0.f || l2_factor != 0.f)) return TTCD_ERR_ARG;
  const bool wide = V > 8192 && rows <= 148LL * (V > 65536 ? 3 : 1);
  auto kern = wide ? ce_rows_kernel<1024> : ce_rows_kernel<256>;
  kern<<<static_cast<unsigned>(rows), wide ? 1024 : 256, 0, static_cast<cudaStream_t>(stream_ptr)>>>(
      static_cast<const bf16*>(logits), static_cast<bf16*>(grad), reinterpret_cast<const int64_t*>(labels), loss_row, lse_row, grad_scale, V, ld,
      ignore_index, write_grad, label_smoothing, lse_square_scale, l2_factor, reinterpret_cast<const float2*>(lse_part),
      n_parts);
  return static_cast<int>(cudaGetLastError());
}

TTCD_EXPORT int ttcd_lse_merge(const void* oa, const float* la, const void* ob, const float* lb, void* out,
                               float* lse_out, long long B, int T, int H, int D, void* stream_ptr) {
  if (D % 2 != 0 || B <= 0) return TTCD_ERR_ARG;
  const long long items = B * T * H;
  lse_merge_kernel<<<static_cast<unsigned>((items + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream_ptr)>>>(
      static_cast<const bf16*>(oa), la, static_cast<const bf16*>(ob), lb, static_cast<bf16*>(out), lse_out, B, T, H, D);
  return static_cast<int>(cudaGetLastError());
}

TTCD_EXPORT int ttcd_adamw(float* p, const void* g, int grad_is_bf16, float* m, float* v, void* p_bf16, long long n,
                           float lr, float beta1, float beta2, float eps, float wd, float bc1, float bc2_sqrt,
                           const float* coef, const int* skip, void* stream_ptr) {
  if (n <= 0) return TTCD_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream_ptr);
  const uintptr_t wide = reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v) |
                         (grad_is_bf16 ? 0 : reinterpret_cast<uintptr_t>(g));
  const uintptr_t narrow = reinterpret_cast<uintptr_t>(p_bf16) | (grad_is_bf16 ? reinterpret_cast<uintptr_t>(g) : 0);
  const bool vec = n >= (128 << 10) && (wide & 15u) == 0 && (narrow & 7u) == 0;
  const unsigned grid = flat_grid(vec ? (n + 3) / 4 : n);
  auto go = [&](auto kern, auto* grad) {
    kern<<<grid, 256, 0, st>>>(p, grad, m, v, static_cast<bf16*>(p_bf16), n, lr, beta1, beta2, eps, wd, bc1, bc2_sqrt, coef, skip);
  };
  if (grad_is_bf16) {
    const bf16* gb = static_cast<const bf16*>(g);
    if (vec) go(adamw_kernel<bf16, true>, gb);
    else go(adamw_kernel<bf16, false>, gb);
  } else {
    const float* gf = static_cast<const float*>(g);
    if (vec) go(adamw_kernel<float, true>, gf);
    else go(adamw_kernel<float, false>, gf);
  }
  return static_cast<int>(cudaGetLastError());
}

// grad, mom fp32 [n], out bf16 [n]; coef, skip: device words or null.
TTCD_EXPORT int ttcd_muon_pre(const float* grad, float* mom, void* out, const float* coef, const int* skip, long long n,
                              float momentum, int nesterov, void* stream_ptr) {
  if (n <= 0) return TTCD_OK;
  const MuonPreParams a{grad, mom, static_cast<bf16*>(out), coef, skip, n, momentum, nesterov};
  const bool vec = n % 4 == 0 && ((reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(mom)) & 15u) == 0 &&
                   (reinterpret_cast<uintptr_t>(out) & 7u) == 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream_ptr);
  if (vec) muon_pre_kernel<4><<<flat_grid(n / 4), 256, 0, st>>>(a);
  else muon_pre_kernel<1><<<flat_grid(n), 256, 0, st>>>(a);
  return static_cast<int>(cudaGetLastError());
}

// u bf16 [n], p fp32 [n], p_bf16 bf16 [n] or null; skip: a device word or null.
TTCD_EXPORT int ttcd_muon_post(const void* u, float* p, void* p_bf16, const int* skip, long long n, float decay, float rate,
                               void* stream_ptr) {
  if (n <= 0) return TTCD_OK;
  const MuonPostParams a{static_cast<const bf16*>(u), p, static_cast<bf16*>(p_bf16), skip, n, decay, rate};
  const bool vec = n % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0 &&
                   ((reinterpret_cast<uintptr_t>(u) | reinterpret_cast<uintptr_t>(p_bf16)) & 7u) == 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream_ptr);
  if (vec) muon_post_kernel<4><<<flat_grid(n / 4), 256, 0, st>>>(a);
  else muon_post_kernel<1><<<flat_grid(n), 256, 0, st>>>(a);
  return static_cast<int>(cudaGetLastError());
}

TTCD_EXPORT int ttcd_sumsq(const void* x, int is_bf16, long long n, float* out, void* stream_ptr) {
  if (n <= 0) return TTCD_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream_ptr);
  if (is_bf16) sumsq_kernel<bf16><<<flat_grid(n), 256, 0, st>>>(static_cast<const bf16*>(x), n, out);
  else sumsq_kernel<float><<<flat_grid(n), 256, 0, st>>>(static_cast<const float*>(x), n, out);
  return static_cast<int>(cudaGetLastError());
}

// kind: 0 bf16->fp32, 1 fp32->bf16, 2 fp32->fp32, 3 bf16->bf16
TTCD_EXPORT int ttcd_cast_scale(const void* x, void* y, long long n, float scale, int kind, int accumulate,
                                void* stream_ptr) {
  if (n <= 0) return TTCD_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream_ptr);
  const unsigned grid = flat_grid(n);
  switch (kind) {
    case 0: cast_scale_kernel<bf16, float><<<grid, 256, 0, st>>>(static_cast<const bf16*>(x), static_cast<float*>(y), n, scale, accumulate); break;
    case 1: cast_scale_kernel<float, bf16><<<grid, 256, 0, st>>>(static_cast<const float*>(x), static_cast<bf16*>(y), n, scale, accumulate); break;
    case 2: cast_scale_kernel<float, float><<<grid, 256, 0, st>>>(static_cast<const float*>(x), static_cast<float*>(y), n, scale, accumulate); break;
    case 3: cast_scale_kernel<bf16, bf16><<<grid, 256, 0, st>>>(static_cast<const bf16*>(x), static_cast<bf16*>(y), n, scale, accumulate); break;
    default: return TTCD_ERR_ARG;
  }
  return static_cast<int>(cudaGetLastError());
}

// y[i] = x[i] * (*factor), bf16, n a multiple of 8, x and y 16-byte aligned; factor: one fp32 on the device.
TTCD_EXPORT int ttcd_scale_by(const void* x, void* y, const float* factor, long long n, void* stream_ptr) {
  if (n <= 0) return TTCD_OK;
  if (n % 8 != 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u)) return TTCD_ERR_ARG;
  const long long blocks = std::min<long long>((n / 8 + 255) / 256, 148LL * 32);
  scale_by_kernel<<<static_cast<unsigned>(blocks), 256, 0, static_cast<cudaStream_t>(stream_ptr)>>>(
      static_cast<const bf16*>(x), static_cast<bf16*>(y), factor, n / 8);
  return static_cast<int>(cudaGetLastError());
}
