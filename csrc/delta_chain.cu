// The chunk-to-chunk chain of the (gated) delta rule (sm_100a; the two products of a step, 64 x D x 32 each, run on the
// tensor cores as TF32 mma.sync tiles with fp32 accumulation: they are far too small for a tcgen05 pipeline; the point
// of the kernel is to run the n dependent steps in ONE launch with the state resident in registers).
//
// For one (batch, head) pair, S [D, Dv] the running state and i the chunk index:
//
//   forward  (i ascending):  states[i] = S;  y_i = x_i - a_i S;          S = gamma_i S + b_i^T y_i
//            a = w (WY factor), b = kt (keys scaled to the chunk end), x = u, y = vn
//   backward (i descending): states[i] = dS; y_i = x_i + a_i dS;         dS = gamma_i dS + add_i - b_i^T y_i
//            a = kt, b = w, x = d_vn (from downstream), add = d_states (from downstream), y = total d_vn
//
// (the role of chunk_gated_delta_rule_fwd_h / chunk_gated_delta_rule_bwd_dhu in fla/ops/common/chunk_delta_h.py).
// The columns of S never mix, so a CTA owns 32 of them (64 for D = 256, where a_i and b_i are large and every column
// slice re-reads them) for the whole sequence: grid (Dv / columns, batch * heads).  Per chunk the CTA stages a_i and
// b_i [64, D] (bf16) in shared memory with asynchronous 16-byte copies that overlap the publication of S.  S [D, columns]
// lives in the accumulator registers of the second product (D / 32 m16n8 tiles per warp) across chunks, in fp32, and is
// mirrored in shared memory, rounded to bf16, as the B operand of the first; y is rounded the same way for the second.
// Every operand of a product is thus a bf16 value (the precision the reference's Triton kernels multiply at), comes to the
// products by ldmatrix and is widened to TF32 there (exactly; bf16 products of 16 would save 10 % of the forward, but sum
// in another order, which a deep model's gradients show), the sums and the state stay fp32.
// The only asynchronous copies are the CTA's own cp.async groups (waited for with wait_group); nothing here waits on
// another CTA, so nothing can spin.
#include "common.cuh"

namespace ttcd {

constexpr int DC_C = 64;         // rows of a chunk
constexpr int DC_THREADS = 256;  // 8 warps

struct DeltaChainParams {
  const bf16* a; const bf16* b;
  const float* gamma; const float* x; const float* add; const float* s_init;
  float* y; float* states; float* s_last;
  int n, D, Dv;
  float sign_a, sign_b;          // y = x + sign_a a S;  S = gamma S + add + sign_b b^T y
  int reverse;
  // optional: per chunk, the sum over this CTA's columns of dot_with[i] * (S entering the step)  ->  dot_out[bh][i][blockIdx.x]
  // (the reverse chain uses it for the gradient of gamma: dot_with = the forward states)
  const float* dot_with; float* dot_out;
};

__device__ __forceinline__ void dc_cp_async16(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void dc_cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void dc_cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void dc_mma8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 of the contraction as two TF32 products of 8 (a bf16 value is an exact TF32 operand after a 16-bit shift).  A register
// of a bf16 fragment holds k = 2 c and 2 c + 1; they take the slots c and c + 4 of both operands.
__device__ __forceinline__ void dc_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  constexpr uint32_t HI = 0xffff0000u;
  dc_mma8(d, a[0] << 16, a[1] << 16, a[0] & HI, a[1] & HI, b0 << 16, b0 & HI);
  dc_mma8(d, a[2] << 16, a[3] << 16, a[2] & HI, a[3] & HI, b1 << 16, b1 & HI);
}
__device__ __forceinline__ void dc_ldm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void dc_ldm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void dc_ldm2t(uint32_t& r0, uint32_t& r1, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}
// B fragments of N8 n-tiles (k x n stored row-wise, `addr` = the lane's address of the first pair) against one A fragment
template <int N8>
__device__ __forceinline__ void dc_load_b(uint32_t (&b)[N8][2], uint32_t addr) {
#pragma unroll
  for (int t = 0; t + 1 < N8; t += 2) {
    uint32_t r[4];
    dc_ldm4t(r, addr + 16 * t);
    b[t][0] = r[0]; b[t][1] = r[1]; b[t + 1][0] = r[2]; b[t + 1][1] = r[3];
  }
  if constexpr (N8 % 2 != 0) dc_ldm2t(b[N8 - 1][0], b[N8 - 1][1], addr + 16 * (N8 - 1));
}

// PIPE: the a / b tiles of the next step travel while this one is computed (two stages of shared memory, fewer CTAs per SM)
template <int D, int DC_COLS, bool PIPE>
__global__ void __launch_bounds__(DC_THREADS, (PIPE ? (D <= 128 ? 2 : 1) : (D <= 128 ? 4 : 2)))
delta_chain_kernel(const DeltaChainParams p) {
  constexpr int LDT = D + 8;                 // bf16 row stride of the a_i / b_i tiles: 16-byte rows, 4 banks apart (ldmatrix)
  constexpr int DC_LDS = DC_COLS + 8;        // bf16 row stride of the [*, columns] tiles read as B operands
  constexpr int NTM = DC_COLS / 8;           // n-tiles per m-tile of S
  constexpr int TPW = (D / 16) * NTM / 8;    // m16n8 tiles of S per warp: tile id = warp * TPW + x -> (id / NTM, id % NTM)
  constexpr int NT = TPW >= NTM ? NTM : TPW; // ... of which NT share an m-tile
  constexpr int MT = TPW / NT;
  constexpr int YT = DC_COLS / 16;           // n-tiles of y per warp
  constexpr int STAGE = 2 * DC_C * LDT;      // bf16 of one (a, b) stage
  extern __shared__ __align__(16) float dc_smem[];
  bf16* stages = reinterpret_cast<bf16*>(dc_smem);          // [1 or 2][a | b][64][LDT]
  bf16* Ss = stages + (PIPE ? 2 : 1) * STAGE;               // [D][columns + 8]   S as the B operand of a S
  bf16* Ys = Ss + D * DC_LDS;                               // [64][columns + 8]  sign_b * y as the B operand of b^T y
  float* red = reinterpret_cast<float*>(Ys + DC_C * DC_LDS);    // [8] per-warp partial sums of the optional dot product
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
  const int col0 = blockIdx.x * DC_COLS;
  const int64_t bh = blockIdx.y;
  const int Dv = p.Dv;
  const bf16* a_base = p.a + bh * p.n * DC_C * D;
  const bf16* b_base = p.b + bh * p.n * DC_C * D;
  const float* x_base = p.x + bh * p.n * DC_C * Dv + col0;
  float* y_base = p.y + bh * p.n * DC_C * Dv + col0;
  float* st_base = p.states + bh * p.n * D * Dv + col0;
  // (only the two-stage form serves the reverse chain)
  const float* add_base = PIPE && p.add != nullptr ? p.add + bh * p.n * D * Dv + col0 : nullptr;
  const float* dot_base = PIPE && p.dot_with != nullptr ? p.dot_with + bh * p.n * D * Dv + col0 : nullptr;
  // the warp's tiles of S: m-tile mt0 + m (rows 16 (mt0 + m) + g, + 8), n-tiles nt0 .. nt0 + NT - 1 (columns 8 nt + 2 c, + 1)
  const int mt0 = (warp * TPW) / NTM, nt0 = (warp * TPW) % NTM;
  // the warp's YT tiles of y: m-tile warp / 2, n-tiles YT (warp % 2) ..
  const int ymt = warp >> 1, ynt0 = YT * (warp & 1);
  // ldmatrix: which 8 x 8 matrix a lane addresses
  const int l8 = lane & 7, hi8 = 8 * ((lane >> 3) & 1), hi16 = 8 * (lane >> 4);
  const uint32_t st_addr = smem_u32(stages), ss_addr = smem_u32(Ss), ys_addr = smem_u32(Ys);
  const uint32_t a_off = 2u * ((16 * ymt + l8 + hi8) * LDT + hi16);                      // a as A (row-wise)
  const uint32_t sb_addr = ss_addr + 2u * ((l8 + hi8) * DC_LDS + 8 * ynt0 + hi16);       // S as B
  const uint32_t b_off = 2u * (DC_C * LDT + (l8 + hi16) * LDT + 16 * mt0 + hi8);         // b^T as A (transposed on load)
  const uint32_t yb_addr = ys_addr + 2u * ((l8 + hi8) * DC_LDS + 8 * nt0 + hi16);        // y as B

  auto load_stage = [&](int step) {
    const int i = p.reverse ? p.n - 1 - step : step;
    const uint4* ga = reinterpret_cast<const uint4*>(a_base + static_cast<int64_t>(i) * DC_C * D);
    const uint4* gb = reinterpret_cast<const uint4*>(b_base + static_cast<int64_t>(i) * DC_C * D);
    const uint32_t dst = st_addr + (PIPE ? (step & 1) * 2u * STAGE : 0u);
#pragma unroll 4
    for (int v = threadIdx.x; v < DC_C * D / 8; v += DC_THREADS) {
      const uint32_t at = dst + 2u * ((v / (D / 8)) * LDT + (v % (D / 8)) * 8);
      dc_cp_async16(at, ga + v);
      dc_cp_async16(at + 2u * DC_C * LDT, gb + v);
    }
    dc_cp_async_commit();
  };
  float2 xv[YT][2];                          // x of the next step's y tiles, in flight
  auto load_x = [&](int step) {
    const int i = p.reverse ? p.n - 1 - step : step;
#pragma unroll
    for (int t = 0; t < YT; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        xv[t][h] = *reinterpret_cast<const float2*>(
            x_base + (static_cast<int64_t>(i) * DC_C + 16 * ymt + g + 8 * h) * Dv + 8 * (ynt0 + t) + 2 * c);
  };
  if (PIPE) load_stage(0);

  float s[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int row = 16 * (mt0 + m) + g, col = 8 * (nt0 + t) + 2 * c;
      const float2 lo = *reinterpret_cast<const float2*>(p.s_init + (bh * D + row) * Dv + col0 + col);
      const float2 hi = *reinterpret_cast<const float2*>(p.s_init + (bh * D + row + 8) * Dv + col0 + col);
      s[m][t][0] = lo.x; s[m][t][1] = lo.y; s[m][t][2] = hi.x; s[m][t][3] = hi.y;
    }
  load_x(0);

  for (int step = 0; step < p.n; ++step) {
    const int i = p.reverse ? p.n - 1 - step : step;
    if (!PIPE) load_stage(step);
    // ---- publish S (to shared memory for the y products, to global memory as states[i])
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const int row = 16 * (mt0 + m) + g, col = 8 * (nt0 + t) + 2 * c;
        const float2 lo = make_float2(s[m][t][0], s[m][t][1]), hi = make_float2(s[m][t][2], s[m][t][3]);
        *reinterpret_cast<__nv_bfloat162*>(Ss + row * DC_LDS + col) = __floats2bfloat162_rn(lo.x, lo.y);      // B operand, rounded once
        *reinterpret_cast<__nv_bfloat162*>(Ss + (row + 8) * DC_LDS + col) = __floats2bfloat162_rn(hi.x, hi.y);
        *reinterpret_cast<float2*>(st_base + (static_cast<int64_t>(i) * D + row) * Dv + col) = lo;
        *reinterpret_cast<float2*>(st_base + (static_cast<int64_t>(i) * D + row + 8) * Dv + col) = hi;
      }
    dc_cp_async_wait_all();
    __syncthreads();
    if (PIPE && step + 1 < p.n) load_stage(step + 1);        // the other stage was last read before this barrier
    const float gm = p.gamma[bh * p.n + i];
    // a tile of the warp's elements of a [D, Dv] tensor of step i: issued a product (or a barrier) before its use
    float ld[MT][NT][4];
    auto load_tile = [&](const float* base) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const int row = 16 * (mt0 + m) + g, col = 8 * (nt0 + t) + 2 * c;
          const float2 lo = *reinterpret_cast<const float2*>(base + (static_cast<int64_t>(i) * D + row) * Dv + col);
          const float2 hi = *reinterpret_cast<const float2*>(base + (static_cast<int64_t>(i) * D + row + 8) * Dv + col);
          ld[m][t][0] = lo.x; ld[m][t][1] = lo.y; ld[m][t][2] = hi.x; ld[m][t][3] = hi.y;
        }
    };
    if (dot_base != nullptr) load_tile(dot_base);
    // ---- y = x + sign_a * (a S): the warp's YT 16 x 8 tiles
    const uint32_t stage = st_addr + (PIPE ? (step & 1) * 2u * STAGE : 0u);
    {
      float acc[YT][4];
#pragma unroll
      for (int t = 0; t < YT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
#pragma unroll 4
      for (int k0 = 0; k0 < D; k0 += 16) {
        uint32_t a[4], b[YT][2];
        dc_ldm4(a, stage + a_off + 2 * k0);
        dc_load_b<YT>(b, sb_addr + 2 * k0 * DC_LDS);
#pragma unroll
        for (int t = 0; t < YT; ++t) dc_mma(acc[t], a, b[t][0], b[t][1]);
      }
#pragma unroll
      for (int t = 0; t < YT; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = 16 * ymt + g + 8 * h, col = 8 * (ynt0 + t) + 2 * c;
          const int64_t off = (static_cast<int64_t>(i) * DC_C + row) * Dv + col;
          const float2 yv = make_float2(xv[t][h].x + p.sign_a * acc[t][2 * h], xv[t][h].y + p.sign_a * acc[t][2 * h + 1]);
          *reinterpret_cast<float2*>(y_base + off) = yv;
          *reinterpret_cast<__nv_bfloat162*>(Ys + row * DC_LDS + col) = __floats2bfloat162_rn(p.sign_b * yv.x, p.sign_b * yv.y);
        }
    }
    if (step + 1 < p.n) load_x(step + 1);
    if (dot_base != nullptr) {
      float part = 0.f;
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
          part += s[m][t][0] * ld[m][t][0] + s[m][t][1] * ld[m][t][1] + s[m][t][2] * ld[m][t][2] + s[m][t][3] * ld[m][t][3];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      if (lane == 0) red[warp] = part;
    }
    // ---- S = gamma S + add + sign_b * (b^T y), accumulated in place; the addend is on its way over the barrier
    if (add_base != nullptr) load_tile(add_base);
    __syncthreads();
    if (dot_base != nullptr && threadIdx.x == 0) {
      float tot = 0.f;
#pragma unroll
      for (int wv = 0; wv < DC_THREADS / 32; ++wv) tot += red[wv];
      p.dot_out[(bh * p.n + i) * (Dv / 32) + blockIdx.x] = tot;        // rows of Dv / 32 slots (zero-filled by the caller)
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[m][t][e] = add_base != nullptr ? fmaf(gm, s[m][t][e], ld[m][t][e]) : gm * s[m][t][e];
#pragma unroll
    for (int k0 = 0; k0 < DC_C; k0 += 16) {
      uint32_t b[NT][2];
      dc_load_b<NT>(b, yb_addr + 2 * k0 * DC_LDS);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[4];
        dc_ldm4t(a, stage + b_off + 2 * (k0 * LDT + 16 * m));
#pragma unroll
        for (int t = 0; t < NT; ++t) dc_mma(s[m][t], a, b[t][0], b[t][1]);
      }
    }
    // (what this step still reads, b and y, is rewritten after the next step's first barrier; PIPE's only stage 0 / 1
    // alternate, a single stage is rewritten at once)
    if (!PIPE) __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const int row = 16 * (mt0 + m) + g, col = 8 * (nt0 + t) + 2 * c;
      *reinterpret_cast<float2*>(p.s_last + (bh * D + row) * Dv + col0 + col) = make_float2(s[m][t][0], s[m][t][1]);
      *reinterpret_cast<float2*>(p.s_last + (bh * D + row + 8) * Dv + col0 + col) = make_float2(s[m][t][2], s[m][t][3]);
    }
}

template <int D, int COLS, bool PIPE>
static int launch_delta_chain(const DeltaChainParams& p, int BH, cudaStream_t stream) {
  constexpr int smem = ((PIPE ? 4 : 2) * DC_C * (D + 8) + D * (COLS + 8) + DC_C * (COLS + 8)) * static_cast<int>(sizeof(bf16)) +
                       8 * static_cast<int>(sizeof(float));
  auto kern = delta_chain_kernel<D, COLS, PIPE>;
  static bool configured = false;
  if (!configured) {
    TTCD_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  kern<<<dim3(p.Dv / COLS, BH), DC_THREADS, smem, stream>>>(p);
  return static_cast<int>(cudaGetLastError());
}

// The chain is a string of dependent steps, so what a step waits for is what it costs.  Two stages of a / b, with the
// addend and the states of the dot product in flight over the products, pay where a CTA has its SM to itself (D = 256,
// at most one CTA per SM) and in the reverse chain, which reads two [D, Dv] tensors more; elsewhere more CTAs per SM hide
// each other's waits.  us (BH x steps, D, Dv), before (scalar 16-bit shared-memory reads, every tile waited for) | now:
// forward 32 x 64, 128, 128: 291 | 179; 12 x 47, 256, 512: 455 | 295; 96 x 64, 256, 512: 2769 | 2045 (one stage);
// reverse, the same: 387 | 240; 720 | 429; 4466 | 3380 (one stage instead of two: 299; 557; 3749).
// The one-stage forms are held to the registers of their CTAs per SM and spill a little: <256, 64> 76 bytes, <64, 32> 28,
// <128, 32> 8 per thread.
template <int D, int COLS>
static int launch_delta_chain(const DeltaChainParams& p, int BH, cudaStream_t stream) {
  const bool alone = D == 256 && static_cast<int64_t>(p.Dv / COLS) * BH <= sm_count();
  if (p.add != nullptr || alone) return launch_delta_chain<D, COLS, true>(p, BH, stream);
  return launch_delta_chain<D, COLS, false>(p, BH, stream);
}

static int delta_chain_dispatch(const DeltaChainParams& p, int BH, cudaStream_t stream) {
  if (BH <= 0 || p.n <= 0 || p.Dv <= 0 || p.Dv % 32 != 0 || BH > 65535) return TTCD_ERR_ARG;
  switch (p.D) {
    case 32: return launch_delta_chain<32, 32>(p, BH, stream);
    case 64: return launch_delta_chain<64, 32>(p, BH, stream);
    case 128: return launch_delta_chain<128, 32>(p, BH, stream);
    case 256: return p.Dv % 64 == 0 ? launch_delta_chain<256, 64>(p, BH, stream) : launch_delta_chain<256, 32>(p, BH, stream);
    default: return TTCD_ERR_ARG;
  }
}

}  // namespace ttcd

// Contiguous tensors: w, kt [BH][n][64][D] bf16; fp32: u, vn [BH][n][64][Dv]; gamma [BH][n]; s0, s_final [BH][D][Dv];
// states [BH][n][D][Dv] (the state entering each chunk).  D in {32, 64, 128, 256}, Dv a multiple of 32.
TTCD_EXPORT int ttcd_delta_chain_fwd(const bf16* w, const float* u, const bf16* kt, const float* gamma, const float* s0,
                                     float* vn, float* states, float* s_final, int BH, int n, int D, int Dv,
                                     void* stream_ptr) {
  ttcd::DeltaChainParams p;
  p.a = w; p.b = kt; p.gamma = gamma; p.x = u; p.add = nullptr; p.s_init = s0;
  p.y = vn; p.states = states; p.s_last = s_final;
  p.n = n; p.D = D; p.Dv = Dv; p.sign_a = -1.f; p.sign_b = 1.f; p.reverse = 0;
  p.dot_with = nullptr; p.dot_out = nullptr;
  return ttcd::delta_chain_dispatch(p, BH, static_cast<cudaStream_t>(stream_ptr));
}

// Reverse chain: d_vn, d_states, d_final are the gradients arriving at vn, states and the final state; writes the total
// gradient of vn (d_vn_tot), the gradient of the state LEAVING each chunk (ds_next [BH][n][D][Dv]) and of s0.  With
// `states` (the forward states) it also writes d_gamma_parts [BH][n][Dv / 32] (zero-filled by the caller): per chunk and
// column slice of a CTA, the sum of states * ds_next (the gradient of the chunk's decay is the sum over a row).
TTCD_EXPORT int ttcd_delta_chain_bwd(const bf16* w, const bf16* kt, const float* gamma, const float* d_vn,
                                     const float* d_states, const float* d_final, float* d_vn_tot, float* ds_next,
                                     float* d_s0, const float* states, float* d_gamma_parts, int BH, int n, int D, int Dv,
                                     void* stream_ptr) {
  ttcd::DeltaChainParams p;
  p.a = kt; p.b = w; p.gamma = gamma; p.x = d_vn; p.add = d_states; p.s_init = d_final;
  p.y = d_vn_tot; p.states = ds_next; p.s_last = d_s0;
  p.n = n; p.D = D; p.Dv = Dv; p.sign_a = 1.f; p.sign_b = -1.f; p.reverse = 1;
  p.dot_with = d_gamma_parts != nullptr ? states : nullptr; p.dot_out = d_gamma_parts;
  return ttcd::delta_chain_dispatch(p, BH, static_cast<cudaStream_t>(stream_ptr));
}
