// y[M, N] = alpha * x[M, K] @ w[N, K]^T for a handful of rows (M <= 16): the decode step, where a 128-row tensor-core
// tile would be almost empty and the op is bound by reading w once.  The reference's decode step
// (custom_models/ipttcd/modeling_ipttcdv9.py forward with a KV cache) runs nn.Linear on one row through the library;
// this is the equivalent for the row counts a decode step has.  What surrounds the product in a decoder layer can ride
// along: RMSNorm of x in front (NORM), SwiGLU of a gate and an up column behind (SWIGLU), a residual added to y.
//
// Work goes in groups of 8 columns of y (8 rows of w; 16 with SWIGLU).  A CTA takes its groups in turn, whole rows at a
// time, through a ring of shared-memory stages filled by asynchronous 16-byte copies, so that its weights stream while
// it computes; its 8 warps split K: w is the B operand of mma.sync m16n8k16 (bf16 x bf16, fp32 accumulation), x the A
// operand (rows beyond M are zero registers; read, and normalised, once per CTA), and the warps' sums meet in shared
// memory in fp32.  Lane (g, c) takes 16 bytes = 8 consecutive k of row g of w and of x; which k a fragment slot stands for
// is free as long as A and B agree, so the 16 bytes serve two MMAs as they are.  The row pitch in shared memory is 64
// bytes more than a multiple of 128, so that eight lanes of two rows hit all banks.
// The kernel may start while the one before it still runs (programmatic dependent launch): the first copies of w are
// issued before it waits for that kernel when the caller says that no kernel still running can be writing w.
//
// us per launch in a graph, weights from HBM (N x K), this kernel: 1 | 8 | 16 rows; in brackets one warp per column with fp32
// FMAs, which one-row calls still take where it is the faster (gemv_row_kernel):
//   4096 x 1024: 4.9 | 4.9 | 6.0 (4.6 | 8.8 | 15);  1024 x 3072: 4.4 | 4.6 | 5.9 (6.4 | 14.5 | 25);
//   2048 x 8192: 11.0 | 13.0 | 20.1 (12.3 | 34 | 63);  16384 x 2048: 15.2 | 15.2 | 16.2 (13.1 | 39 | 71);
//   151936 x 1024: 49 | 51 | 72 (47 | 175 | 338);  128256 x 2048: 82 | 84 | 92 (76 | 264 | 513).
// Where two CTAs share an SM (up to 8 rows), groups of 16 rows of w (SwiGLU, or a wide output) leave a CTA's ring one stage
// beyond K = 1568 (a stage of K = 2048 is 66 KB): nothing of it is in flight while it computes, only the other CTA reads.  The
// wide output is at 6.4 TB/s all the same; SwiGLU of 8192 x 2048 takes 13.9 us (67 MB).
#include "common.cuh"

#include <algorithm>

namespace ttcd {

constexpr int GV_WARPS = 8;
constexpr int GV_NORM_K = 2048;    // NORM needs the warps' whole shares of x in registers

struct GemvParams {
  const bf16* x; const bf16* w; bf16* y;
  const bf16* res;                 // optional [M, N]: y = bf16(product) + res
  const bf16* norm_w;              // NORM: weight [K]
  int M, N, K;                     // SWIGLU: N columns of y; w has 2 N rows, gate then up
  int64_t ldx, ldw, ldy, ldres;
  float alpha, eps;
  int early_w;                     // w may be read before the previous kernel has finished
};

__device__ __forceinline__ void gv_cp_async16(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void gv_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float gv_sumsq(const uint4& v) {
  const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), c = unpack_bf16(v.z), d = unpack_bf16(v.w);
  return a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + c.x * c.x + c.y * c.y + d.x * d.x + d.y * d.y;
}
__device__ __forceinline__ uint32_t gv_norm2(uint32_t x, uint32_t w, float r) {
  const float2 a = unpack_bf16(x), b = unpack_bf16(w);
  return pack_bf16(a.x * r * b.x, a.y * r * b.y);
}
__host__ __device__ constexpr int gv_pitch(int kc) { return kc * 2 + ((64 - (kc * 2) % 128) + 128) % 128; }      // bytes

__host__ __device__ constexpr int gv_xs(bool hi, bool norm) { return hi || norm ? 8 : 12; }
__host__ __device__ constexpr int gv_slots(bool hi) { return 148 * (hi ? 1 : 2); }      // CTAs that run at once
template <int N>
__device__ __forceinline__ void gv_cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// HI: rows 8 .. 15 of x exist.  WIDE: groups of 16 columns.  STAGES: depth of the ring.
template <bool HI, bool SWIGLU, bool NORM, bool WIDE, int STAGES>
__global__ void __launch_bounds__(GV_WARPS * 32, (HI ? 1 : 2)) gemv_small_kernel(const GemvParams p) {
  static_assert(!(SWIGLU && WIDE), "one or the other");
  constexpr int T = SWIGLU || WIDE ? 2 : 1;                // n-tiles of 8 rows of w per group
  constexpr int ROWS = 8 * T, COLS = WIDE ? 16 : 8;        // rows of w, columns of y per group
  constexpr int XS = gv_xs(HI, NORM);                         // 32-wide k steps of x a warp holds in registers
  constexpr int KC = XS * 32 * GV_WARPS;                   // columns of w in a stage
  extern __shared__ __align__(16) uint8_t gv_smem[];
  __shared__ float part[GV_WARPS][T][16][8];
  __shared__ float ssum[GV_WARPS][16];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  const int groups = (p.N + COLS - 1) / COLS, chunks = (p.K + KC - 1) / KC;
  const int mine = (groups - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
  const int items = mine * chunks;                         // (group, chunk of K) pairs, chunk fastest
  const int pitch = gv_pitch(min(p.K, KC)), stage_bytes = ROWS * pitch;
  const uint32_t sbase = smem_u32(gv_smem);
  // row r of a group: column COLS group + r of y (SWIGLU: r - 8 for the up half); columns past N re-read the last one.
  // Called for items 0, 1, 2, ... in turn: the next one's group, chunk and stage are counted, not divided for.
  int next = 0, next_n0 = static_cast<int>(blockIdx.x) * COLS, next_ch = 0, next_stage = 0;
  auto load_next = [&]() {
    if (next < items) {
      const int kc0 = next_ch * KC, vecs = min(KC, p.K - kc0) / 8;
      const uint32_t dst = sbase + next_stage * stage_bytes;
#pragma unroll
      for (int r = warp; r < ROWS; r += GV_WARPS) {
        const int col = SWIGLU ? min(next_n0 + (r & 7), p.N - 1) + (r >= 8 ? p.N : 0) : min(next_n0 + r, p.N - 1);
        const bf16* src = p.w + static_cast<int64_t>(col) * p.ldw + kc0;
#pragma unroll 4
        for (int v = lane; v < vecs; v += 32) gv_cp_async16(dst + r * pitch + v * 16, src + v * 8);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");   // (an empty group keeps the count)
    ++next;
    if (++next_stage == STAGES) next_stage = 0;
    if (++next_ch == chunks) { next_ch = 0; next_n0 += static_cast<int>(gridDim.x) * COLS; }
  };
  auto fill = [&]() {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) load_next();
  };
  if (p.early_w) fill();
  pdl_wait();
  pdl_launch_dependents();
  if (!p.early_w) fill();

  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const bf16* x0 = p.x + static_cast<int64_t>(g < p.M ? g : 0) * p.ldx;
  const bf16* x1 = p.x + static_cast<int64_t>(HI && g + 8 < p.M ? g + 8 : 0) * p.ldx;
  uint4 a[XS], h[HI ? XS : 1];
  int k_lo = 0, k_hi = 0, per = 0;
  // this warp's share of chunk `ch` of x
  auto load_x = [&](int ch) {
    const int kc0 = ch * KC, kc = min(KC, p.K - kc0);
    per = ((kc + 31) / 32 + GV_WARPS - 1) / GV_WARPS;
    k_lo = warp * per * 32;
    k_hi = min(kc, k_lo + per * 32);
#pragma unroll
    for (int u = 0; u < XS; ++u) {                         // K is a multiple of 8: a lane's 8 values all exist or none does
      const int k = k_lo + 32 * u + 8 * c;
      a[u] = g < p.M && k < k_hi ? *reinterpret_cast<const uint4*>(x0 + kc0 + k) : zero;
      if (HI) h[u] = g + 8 < p.M && k < k_hi ? *reinterpret_cast<const uint4*>(x1 + kc0 + k) : zero;
    }
  };
  load_x(0);
  if constexpr (NORM) {                                    // one chunk: K <= GV_NORM_K
    float q0 = 0.f, q1 = 0.f;
#pragma unroll
    for (int u = 0; u < XS; ++u) {
      q0 += gv_sumsq(a[u]);
      if (HI) q1 += gv_sumsq(h[u]);
    }
    q0 += __shfl_xor_sync(0xffffffffu, q0, 1); q0 += __shfl_xor_sync(0xffffffffu, q0, 2);
    q1 += __shfl_xor_sync(0xffffffffu, q1, 1); q1 += __shfl_xor_sync(0xffffffffu, q1, 2);
    if (c == 0) { ssum[warp][g] = q0; ssum[warp][g + 8] = q1; }
    __syncthreads();
    float t0 = 0.f, t1 = 0.f;
#pragma unroll
    for (int w = 0; w < GV_WARPS; ++w) { t0 += ssum[w][g]; if (HI) t1 += ssum[w][g + 8]; }
    const float r0 = rsqrtf(t0 / p.K + p.eps), r1 = HI ? rsqrtf(t1 / p.K + p.eps) : 0.f;
#pragma unroll
    for (int u = 0; u < XS; ++u) {
      const int k = k_lo + 32 * u + 8 * c;
      const uint4 nw = k < k_hi ? *reinterpret_cast<const uint4*>(p.norm_w + k) : zero;
      a[u] = make_uint4(gv_norm2(a[u].x, nw.x, r0), gv_norm2(a[u].y, nw.y, r0), gv_norm2(a[u].z, nw.z, r0), gv_norm2(a[u].w, nw.w, r0));
      if (HI)
        h[u] = make_uint4(gv_norm2(h[u].x, nw.x, r1), gv_norm2(h[u].y, nw.y, r1), gv_norm2(h[u].z, nw.z, r1), gv_norm2(h[u].w, nw.w, r1));
    }
  }

  float acc[T][4];
  int ch = 0, stage = 0, n0 = static_cast<int>(blockIdx.x) * COLS;
  for (int it = 0; it < items; ++it) {
    if (ch == 0) {
#pragma unroll
      for (int t = 0; t < T; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    }
    if (!NORM && chunks > 1 && it > 0) load_x(ch);
    gv_cp_async_wait<STAGES - 1>();
    __syncthreads();
    const uint8_t* ws = gv_smem + stage * stage_bytes;
    if (++stage == STAGES) stage = 0;
#pragma unroll
    for (int u = 0; u < XS; ++u) {
      if (u < per) {
        const int k = k_lo + 32 * u + 8 * c;
#pragma unroll
        for (int t = 0; t < T; ++t) {
          const uint4 b = k < k_hi ? *reinterpret_cast<const uint4*>(ws + (g + 8 * t) * pitch + k * 2) : zero;
          gv_mma(acc[t], a[u].x, HI ? h[u].x : 0u, a[u].y, HI ? h[u].y : 0u, b.x, b.y);
          gv_mma(acc[t], a[u].z, HI ? h[u].z : 0u, a[u].w, HI ? h[u].w : 0u, b.z, b.w);
        }
      }
    }
    const bool last = ch == chunks - 1;
    if (last) {                                            // rows g, g + 8 of y, columns 2 c, + 1 of the group
#pragma unroll
      for (int t = 0; t < T; ++t) {
        *reinterpret_cast<float2*>(&part[warp][t][g][2 * c]) = make_float2(acc[t][0], acc[t][1]);
        if (HI) *reinterpret_cast<float2*>(&part[warp][t][g + 8][2 * c]) = make_float2(acc[t][2], acc[t][3]);
      }
    }
    __syncthreads();                                       // the stage is free, the partial sums are there
    load_next();
    if (last) {
      if (static_cast<int>(threadIdx.x) < p.M * COLS) {
        const int col = threadIdx.x % COLS, m = threadIdx.x / COLS, n = n0 + col;
        if (n < p.N) {
          float v = 0.f;
#pragma unroll
          for (int w = 0; w < GV_WARPS; ++w) v += part[w][WIDE ? col >> 3 : 0][m][col & 7];
          bf16 out = __float2bfloat16(v * p.alpha);
          if constexpr (SWIGLU) {
            float u = 0.f;
#pragma unroll
            for (int w = 0; w < GV_WARPS; ++w) u += part[w][T - 1][m][col];
            const float gate = __bfloat162float(out), up = __bfloat162float(__float2bfloat16(u * p.alpha));
            out = __float2bfloat16(gate / (1.f + __expf(-gate)) * up);
          }
          if (p.res != nullptr) out = __float2bfloat16(__bfloat162float(out) + __bfloat162float(p.res[m * p.ldres + n]));
          p.y[m * p.ldy + n] = out;
        }
      }
      ch = 0;
      n0 += static_cast<int>(gridDim.x) * COLS;
    } else {
      ++ch;
    }
    // (the next item's partial sums are written after its first barrier)
  }
}

// One row of x and nothing riding along: a warp per column of y, fp32 FMAs, x through L1; no ring to fill, no barrier between
// groups.  Where a CTA of the kernel above has more than one group (N > 8 x 296) and K fills the warps' loads of 256.
// us, this | the kernel above: 4096 x 1024: 4.6 | 5.0, 8192 x 1024: 5.8 | 8.0, 16384 x 2048: 13.1 | 15.2, 128256 x 2048: 76 |
// 82;  2048 x 2048: 5.5 | 4.5, 1024 x 3072: 6.4 | 4.4, 49152 x 960: 25.4 | 20.2.
__global__ void __launch_bounds__(256) gemv_row_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, bf16* __restrict__ y,
                                                       int N, int K, int64_t ldw, float alpha) {
  const int lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (n >= N) return;
  float acc = 0.f;
  const bf16* wr = w + static_cast<int64_t>(n) * ldw;
  for (int k = lane * 8; k < K; k += 256) {
    const uint4 wv = *reinterpret_cast<const uint4*>(wr + k), xv = *reinterpret_cast<const uint4*>(x + k);
    const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w}, xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = unpack_bf16(ww[i]), b = unpack_bf16(xw[i]);
      acc = fmaf(a.x, b.x, fmaf(a.y, b.y, acc));
    }
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane == 0) y[n] = __float2bfloat16(acc * alpha);
}

template <bool HI, bool SWIGLU, bool NORM, bool WIDE, int STAGES>
static int launch_gemv(const GemvParams& p, int smem, cudaStream_t stream) {
  auto kern = gemv_small_kernel<HI, SWIGLU, NORM, WIDE, STAGES>;
  static bool configured = false;
  if (!configured) {
    TTCD_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    configured = true;
  }
  // equal turns: as many CTAs as run at once at most, each with the same number of groups (the last ones one less)
  constexpr int cols = WIDE ? 16 : 8;
  const int groups = (p.N + cols - 1) / cols, slots = gv_slots(HI), turns = (groups + slots - 1) / slots;
  return launch_dependent(kern, dim3((groups + turns - 1) / turns), dim3(GV_WARPS * 32), smem, stream, p);
}

template <bool HI, bool SWIGLU, bool NORM, bool WIDE>
static int stages_gemv(const GemvParams& p, cudaStream_t stream) {
  constexpr int KC = gv_xs(HI, NORM) * 32 * GV_WARPS;
  const int stage = (SWIGLU || WIDE ? 16 : 8) * gv_pitch(std::min(p.K, KC));
  // as deep a ring as the CTAs of an SM have room for: two, or one with more than 8 rows (a stage is at most 99 KB)
  constexpr int room = (HI ? 200 : 100) * 1024;
  if (4 * stage <= room) return launch_gemv<HI, SWIGLU, NORM, WIDE, 4>(p, 4 * stage, stream);
  if (3 * stage <= room) return launch_gemv<HI, SWIGLU, NORM, WIDE, 3>(p, 3 * stage, stream);
  if (2 * stage <= room) return launch_gemv<HI, SWIGLU, NORM, WIDE, 2>(p, 2 * stage, stream);
  return launch_gemv<HI, SWIGLU, NORM, WIDE, 1>(p, stage, stream);
}

template <bool HI, bool SWIGLU, bool NORM>
static int dispatch_gemv(const GemvParams& p, cudaStream_t stream) {
  // many turns per CTA (an output vocabulary): twice the columns per turn halve the barriers (151936 x 1024, one row: 78 -> 50 us,
  // 6.2 TB/s; 128256 x 2048: 82 us, 6.4 TB/s, with a ring of one stage)
  if constexpr (!SWIGLU) {
    if (p.N >= 4 * 8 * gv_slots(HI) && p.K <= 2048) return stages_gemv<HI, SWIGLU, NORM, true>(p, stream);
  }
  return stages_gemv<HI, SWIGLU, NORM, false>(p, stream);
}

}  // namespace ttcd

// x: [M, K] bf16 rows ldx apart, w: [N, K] bf16 rows ldw apart, y: [M, N] bf16; 1 <= M <= 16, K a multiple of 8,
// x / w 16-byte aligned with ldx, ldw multiples of 8.
//   res (may be null): [M, N] bf16 rows ldres apart, added to the rounded product (the sum is rounded again).
//   norm_w (may be null): [K] bf16, 16-byte aligned: x is RMS-normalised first (eps), K <= 2048.
//   swiglu: w is [2 N, K], gate rows then up rows; y = silu(gate) * up of the rounded products.
//   early_w: the caller knows that no kernel that may still be running writes w.
TTCD_EXPORT int ttcd_gemv_small(const void* x, const void* w, void* y, const void* res, const void* norm_w, int M, int N,
                                int K, long long ldx, long long ldw, long long ldy, long long ldres, float alpha, float eps,
                                int swiglu, int early_w, void* stream_ptr) {
  using namespace ttcd;
  if (M < 1 || M > 16 || N < 1 || K < 8 || K % 8 != 0 || ldx % 8 != 0 || ldw % 8 != 0) return TTCD_ERR_ARG;
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(norm_w)) & 15u))
    return TTCD_ERR_ARG;
  if (norm_w != nullptr && K > GV_NORM_K) return TTCD_ERR_ARG;
  GemvParams p;
  p.x = static_cast<const bf16*>(x); p.w = static_cast<const bf16*>(w); p.y = static_cast<bf16*>(y);
  p.res = static_cast<const bf16*>(res); p.norm_w = static_cast<const bf16*>(norm_w);
  p.M = M; p.N = N; p.K = K;
  p.ldx = ldx; p.ldw = ldw; p.ldy = ldy; p.ldres = ldres;
  p.alpha = alpha; p.eps = eps; p.early_w = early_w;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const bool norm = norm_w != nullptr;
  if (M == 1 && !norm && !swiglu && res == nullptr && !early_w && N > 8 * gv_slots(false) && (K % 256 == 0 || K < 256)) {
    gemv_row_kernel<<<static_cast<unsigned>((N + 7) / 8), 256, 0, stream>>>(p.x, p.w, p.y, N, K, ldw, alpha);
    return static_cast<int>(cudaGetLastError());
  }
  if (M > 8) {
    if (swiglu) return norm ? dispatch_gemv<true, true, true>(p, stream) : dispatch_gemv<true, true, false>(p, stream);
    return norm ? dispatch_gemv<true, false, true>(p, stream) : dispatch_gemv<true, false, false>(p, stream);
  }
  if (swiglu) return norm ? dispatch_gemv<false, true, true>(p, stream) : dispatch_gemv<false, true, false>(p, stream);
  return norm ? dispatch_gemv<false, false, true>(p, stream) : dispatch_gemv<false, false, false>(p, stream);
}
