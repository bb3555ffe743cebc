// Persistent, warp-specialised bf16 GEMM for sm_100a.
//
//   C[b][m][n] = alpha * rowscale[m] * sum_k A[b][m][k] * B[b][n][k]  (+ beta * Cin[b][m][n])
//
// A is given either K-major ([M, K] row-major) or MN-major ([K, M] row-major); likewise B
// ([N, K] or [K, N]).  That covers y = x W^T, dx = dy W, dW = dy^T x and their batched forms
// without any transposition pass.
//
// One CTA per SM; tile 128 x BN x 64 (BN 256, 128 or 64: see gemm_tile_n).  Warp 0 streams operand tiles with TMA (128-byte swizzle,
// no multicast) through a mbarrier ring of 4 to 8 stages, one thread of warp 1 issues tcgen05.mma into a
// double-buffered TMEM accumulator (2 x BN fp32 columns), warps 2-5 drain the other accumulator
// with tcgen05.ld and write C, so the epilogue of tile i overlaps the main loop of tile i+1.
// Replaces the reference's cuBLAS calls behind nn.Linear / torch.matmul
// (custom_models/ipttcd/modeling_ipttcdv9_lowcopy_scanfuse.py:113-200).
#include "gemm.cuh"

namespace ttcd {

constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;
// warps that drain an accumulator: four, or with SwiGLU one per 32 lanes and 32 columns of C (four of them take 22 k cycles for what the
// MMAs of a 1024-long product make in 8 k: exponential, division and a dependent chain per value)
__host__ __device__ constexpr int gemm_epi_warps(int bn, bool swiglu) { return swiglu ? bn / 16 : 4; }
__host__ __device__ constexpr int gemm_threads(int bn, bool swiglu) { return 64 + 32 * gemm_epi_warps(bn, swiglu); }

struct GemmParams {
  int64_t M, N, K, batch;
  int64_t ldc, stride_c;     // elements
  int64_t tiles_m, tiles_n;  // per batch
  float alpha, beta;
  const bf16* row_scale;     // optional [batch*M]
  int a_bcast, b_bcast;      // operand shared by every batch entry (its tensor map has batch 1)
  int accumulate;            // fp32 output: add to C in memory (C is the addend: beta = 1, Cin = C) instead of storing
  int m_fastest;             // raster order inside a batch entry: consecutive tiles walk M (the B panel is the big one)
  float2* lse_part;          // optional [batch*M][tiles_n]: per row and column tile (max, sum of exp(x - max)) of the
                             // bf16-rounded outputs, for a log-sum-exp over the row without another pass (bf16 out only)
  int64_t seg1, seg2;        // first column of the second and third matrix that B's rows come from (past the last: there is none)
  int round_first;           // the product is rounded to bf16 before Cin is added
};
struct GemmBMaps { CUtensorMap m[3]; };

template <int BN, int STAGES>
struct GemmSmem {
  static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;
  static constexpr int B_BYTES = BN * GEMM_BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  // epilogue staging for TMA stores: 4 warps x 2 buffers x (32 rows x 128 bytes), 128-byte swizzled
  static constexpr int EPI_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int EPI_BYTES = 4 * 2 * 4096;
  static constexpr int BAR_OFFSET = EPI_OFFSET + EPI_BYTES;
  // full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], tmem base word, abort flag
  static constexpr int TOTAL = BAR_OFFSET + (2 * STAGES + 4) * 8 + 16;
};

// Whether `ok` holds for every thread of the two warps that meet at named barrier `bar`.
__device__ __forceinline__ bool pair_all(bool ok, int bar) {
  uint32_t all;
  __syncwarp();
  asm volatile(
      "{\n\t.reg .pred P, Q;\n\t"
      "setp.ne.b32 P, %1, 0;\n\t"
      "bar.red.and.pred Q, %2, 64, P;\n\t"
      "selp.u32 %0, 1, 0, Q;\n\t}"
      : "=r"(all)
      : "r"(static_cast<uint32_t>(ok)), "r"(bar)
      : "memory");
  return all != 0;
}

// SWIGLU: B's rows are half gate, half up; a tile of BN rows of B makes BN / 2 columns of C.  The product never reaches memory:
// gate | up of 65536 x 3072 (K 1024) and the pass that combined them took 600 + 250 us, with 1.6 GB between them; 585 us so.
template <int BN, int STAGES, bool A_MN, bool B_MN, typename OutT, bool HAS_CIN, bool SWIGLU = false>
__global__ void __launch_bounds__(gemm_threads(BN, SWIGLU), 1)
gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ GemmBMaps tma_bs,
            const __grid_constant__ CUtensorMap tma_c, OutT* __restrict__ C, const OutT* __restrict__ Cin,
            const GemmParams p) {
  using S = GemmSmem<BN, STAGES>;
  constexpr int CN = SWIGLU ? BN / 2 : BN;         // columns of C per tile
  static_assert(!SWIGLU || (!A_MN && !B_MN && !HAS_CIN && sizeof(OutT) == 2), "inference product");
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment: required by the 128-byte swizzle pattern shared by TMA and UMMA.
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_base + S::BAR_OFFSET;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * STAGES + 2 + b); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + S::BAR_OFFSET + (2 * STAGES + 4) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  constexpr uint32_t TMEM_COLS = 2 * BN;  // 128, 256 or 512: power of two

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull_bar(b), 1);
      mbar_init(tempty_bar(b), gemm_epi_warps(BN, SWIGLU));  // one arrival per epilogue warp
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tma_a);
    tma_prefetch_desc(&tma_bs.m[0]);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  pdl_wait();                                      // (what is above touches nothing that the kernel before may write)
  __syncthreads();
  pdl_launch_dependents();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int64_t tiles_per_batch = p.tiles_m * p.tiles_n;
  const int64_t total_tiles = tiles_per_batch * p.batch;
  const int num_kb = static_cast<int>((p.K + GEMM_BK - 1) / GEMM_BK);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        const int b = static_cast<int>(tile / tiles_per_batch);
        const int64_t r = tile % tiles_per_batch;
        const int m0 = static_cast<int>(p.m_fastest ? r % p.tiles_m : r / p.tiles_n) * GEMM_BM;
        int n0 = static_cast<int>(p.m_fastest ? r / p.tiles_m : r % p.tiles_n) * CN;
        const int seg = SWIGLU ? 0 : (n0 >= p.seg1) + (n0 >= p.seg2);      // (a tile lies in one of them)
        const CUtensorMap* tma_b = &tma_bs.m[seg];
        if (seg > 0) n0 -= static_cast<int>(seg == 1 ? p.seg1 : p.seg2);
        const int za = p.a_bcast ? 0 : b, zb = p.b_bcast ? 0 : b;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, 101)) { ok = false; break; }
          const uint32_t sa = smem_base + stage * S::STAGE_BYTES;
          const uint32_t sb = sa + S::A_BYTES;
          mbar_expect_tx(full_bar(stage), S::STAGE_BYTES);
          const int k0 = kb * GEMM_BK;
          if (!A_MN) {
            tma_load_3d(sa, &tma_a, full_bar(stage), k0, m0, za);
          } else {
#pragma unroll
            for (int h = 0; h < GEMM_BM / 64; ++h)
              tma_load_3d(sa + h * (GEMM_BK * 128), &tma_a, full_bar(stage), m0 + h * 64, k0, za);
          }
          if constexpr (SWIGLU) {
            tma_load_3d(sb, &tma_bs.m[0], full_bar(stage), k0, n0, zb);
            tma_load_3d(sb + CN * 128, &tma_bs.m[1], full_bar(stage), k0, n0, zb);
          } else if (!B_MN) {
            tma_load_3d(sb, tma_b, full_bar(stage), k0, n0, zb);
          } else {
#pragma unroll
            for (int h = 0; h < BN / 64; ++h)
              tma_load_3d(sb + h * (GEMM_BK * 128), tma_b, full_bar(stage), n0 + h * 64, k0, zb);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        // abort path: give copies already in flight a bounded time to land before smem is released
        for (int s = 0; s < STAGES; ++s) mbar_drain(full_bar(s), 0), mbar_drain(full_bar(s), 1);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(GEMM_BM, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t acc_phase[2] = {0, 0};
      int acc = 0;
      bool ok = true;
      for (int64_t tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        if (!mbar_wait(tempty_bar(acc), acc_phase[acc] ^ 1u, abort_flag, 102)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, 103)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_base + stage * S::STAGE_BYTES;
          const uint32_t sb = sa + S::A_BYTES;
#pragma unroll
          for (int k = 0; k < GEMM_BK / 16; ++k) {
            // K-major: 16 k-elements = 32 bytes inside the swizzled row; MN-major: 16 k-rows = 2 KiB.
            const uint64_t ad = A_MN ? umma_desc_sw128(sa + k * 2048, GEMM_BK * 128, 1024)
                                     : umma_desc_sw128(sa + k * 32, 16, 1024);
            const uint64_t bd = B_MN ? umma_desc_sw128(sb + k * 2048, GEMM_BK * 128, 1024)
                                     : umma_desc_sw128(sb + k * 32, 16, 1024);
            umma_ss(d_tmem, ad, bd, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(empty_bar(stage));  // frees the smem stage when these MMAs retire
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit(tfull_bar(acc));  // accumulator complete
        acc_phase[acc] ^= 1u;
        acc ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..)
    const int quarter = warp & 3;  // TMEM lane quarter this warp may access
    uint32_t acc_phase[2] = {0, 0};
    int acc = 0;
    // stores of this warp so far: the two staging buffers take turns over the tiles too.  (Counted anew in each tile, a tile with an odd
    // number of stores, 64 columns wide or cut at the edge, left its last store on the buffer that the next tile writes first.)
    int stores = 0;
    bool ok = true;
    for (int64_t tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
      const int b = static_cast<int>(tile / tiles_per_batch);
      const int64_t r = tile % tiles_per_batch;
      const int64_t m0 = (p.m_fastest ? r % p.tiles_m : r / p.tiles_n) * GEMM_BM;
      const int64_t n0 = (p.m_fastest ? r / p.tiles_m : r % p.tiles_n) * CN;
      // With SwiGLU a warp and its neighbour fill one box: 32 columns each, of 64.
      const int part = (warp - 2) >> 2, pair = part >> 1, pair_bar = 1 + quarter * 2 + pair;
      ok = mbar_wait(tfull_bar(acc), acc_phase[acc], abort_flag, 104);
      if constexpr (SWIGLU) {
        if ((part & 1) == 0 && lane == 0) tma_store_wait_read0();     // the last tile's store has released the buffer
        // The two go on or leave together: one that left alone would keep the other at their next barrier for good.
        ok = pair_all(ok, pair_bar);
      }
      if (!ok) break;
      tc_fence_after_sync();
      const int64_t row = m0 + quarter * 32 + lane;
      const bool row_ok = row < p.M;
      float rs = p.alpha;
      if (p.row_scale != nullptr && row_ok) rs *= __bfloat162float(p.row_scale[b * p.M + row]);
      OutT* crow = C + b * p.stride_c + row * p.ldc;
      const OutT* cin_row = HAS_CIN ? (Cin + b * p.stride_c + row * p.ldc) : nullptr;
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * BN;
      if constexpr (SWIGLU) {
        const int c = part * 32;
        uint8_t* buf = smem + S::EPI_OFFSET + quarter * 8192 + pair * 4096;
        uint32_t vg[32], vu[32];
        tmem_ld32(t_row + c, vg);
        tmem_ld32(t_row + CN + c, vu);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty_bar(acc));      // the accumulator is in registers
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          float o[8];
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float2 gate = unpack_bf16(pack_bf16(__uint_as_float(vg[j + e]) * rs, __uint_as_float(vg[j + e + 1]) * rs));
            const float2 up = unpack_bf16(pack_bf16(__uint_as_float(vu[j + e]) * rs, __uint_as_float(vu[j + e + 1]) * rs));
            o[e] = gate.x / (1.f + __expf(-gate.x)) * up.x;
            o[e + 1] = gate.y / (1.f + __expf(-gate.y)) * up.y;
          }
          uint4 w;
          w.x = pack_bf16(o[0], o[1]);
          w.y = pack_bf16(o[2], o[3]);
          w.z = pack_bf16(o[4], o[5]);
          w.w = pack_bf16(o[6], o[7]);
          *reinterpret_cast<uint4*>(buf + sw128_offset(lane, (c & 32) / 8 + (j >> 3))) = w;
        }
        fence_proxy_async_smem();
        asm volatile("bar.sync %0, 64;" ::"r"(pair_bar) : "memory");
        const int64_t col = n0 + pair * 64;
        if ((part & 1) == 0 && lane == 0 && col < p.N) {
          tma_store_3d(&tma_c, smem_u32(buf), static_cast<int>(col), static_cast<int>(m0 + quarter * 32), b);
          tma_store_commit();
        }
        acc_phase[acc] ^= 1u;
        acc ^= 1;
        continue;
      } else if constexpr (sizeof(OutT) == 2) {
        // bf16 output: TMEM -> registers -> swizzled shared memory -> TMA store of a 32-row x 64-column box
        // (full 128-byte lines, clipped at the matrix edges by the tensor map); two staging buffers per warp.
        uint8_t* stage = smem + S::EPI_OFFSET + quarter * 8192;
        const bool want_lse = p.lse_part != nullptr;
        float run_m = -INFINITY, run_s = 0.f;
#pragma unroll 1
        for (int c = 0; c < BN; c += 64, ++stores) {
          const int64_t col = n0 + c;
          if (col >= p.N) break;                      // nothing of this box is in C: no store, no turn
          uint32_t v0[32], v1[32];
          tmem_ld32(t_row + c, v0);
          tmem_ld32(t_row + c + 32, v1);
          if (lane == 0) tma_store_wait_read1();      // the store issued two chunks ago has released this buffer
          __syncwarp();
          tmem_ld_wait();
          uint8_t* buf = stage + (stores & 1) * 4096;
#pragma unroll
          for (int j = 0; j < 64; j += 8) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(j < 32 ? v0[(j & 31) + e] : v1[(j & 31) + e]) * rs;
            if constexpr (HAS_CIN) {
              if (p.round_first) {
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                  const float2 t = unpack_bf16(pack_bf16(f[e], f[e + 1]));
                  f[e] = t.x; f[e + 1] = t.y;
                }
              }
              if (row_ok && col + j + 8 <= p.N) {
                const uint4 cv = *reinterpret_cast<const uint4*>(cin_row + col + j);
                const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 t = unpack_bf16(cw[e]);
                  f[2 * e] += p.beta * t.x;
                  f[2 * e + 1] += p.beta * t.y;
                }
              } else if (row_ok) {
                for (int e = 0; e < 8 && col + j + e < p.N; ++e) f[e] += p.beta * __bfloat162float(cin_row[col + j + e]);
              }
            }
            uint4 o;
            o.x = pack_bf16(f[0], f[1]);
            o.y = pack_bf16(f[2], f[3]);
            o.z = pack_bf16(f[4], f[5]);
            o.w = pack_bf16(f[6], f[7]);
            *reinterpret_cast<uint4*>(buf + sw128_offset(lane, j >> 3)) = o;
            if (want_lse) {
              // running (max, sum) over this thread's row, on the values as the consumer will read them (bf16)
              const uint32_t ow[4] = {o.x, o.y, o.z, o.w};
              float r[8];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float2 t = unpack_bf16(ow[e]);
                r[2 * e] = col + j + 2 * e < p.N ? t.x : -INFINITY;
                r[2 * e + 1] = col + j + 2 * e + 1 < p.N ? t.y : -INFINITY;
              }
              float mx = r[0];
#pragma unroll
              for (int e = 1; e < 8; ++e) mx = fmaxf(mx, r[e]);
              if (mx > run_m) {
                run_s *= __expf(run_m - mx);
                run_m = mx;
              }
              if (run_m != -INFINITY) {
#pragma unroll
                for (int e = 0; e < 8; ++e) run_s += __expf(r[e] - run_m);
              }
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tma_c, smem_u32(buf), static_cast<int>(col), static_cast<int>(m0 + quarter * 32), b);
            tma_store_commit();
          }
        }
        if (want_lse && row_ok) p.lse_part[(b * p.M + row) * p.tiles_n + n0 / BN] = make_float2(run_m, run_s);
      } else if constexpr (!HAS_CIN) {
        // fp32 output: the same way, in boxes of 32 rows x 32 columns.  A thread owns a row, so plain stores would
        // touch 32 lines per instruction with 16 bytes each.  `accumulate` adds the box to C in the L2 instead of
        // reading C into the epilogue: lm_head weight gradient of 640 rows (128256 x 2048, K 640): 1.36 ms before.
        uint8_t* stage = smem + S::EPI_OFFSET + quarter * 8192;
#pragma unroll 1
        for (int c = 0; c < BN; c += 32, ++stores) {
          const int64_t col = n0 + c;
          if (col >= p.N) break;
          uint32_t v[32];
          tmem_ld32(t_row + c, v);
          if (lane == 0) tma_store_wait_read1();      // the store issued two chunks ago has released this buffer
          __syncwarp();
          tmem_ld_wait();
          uint8_t* buf = stage + (stores & 1) * 4096;
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            float4 o;
            o.x = __uint_as_float(v[j]) * rs;
            o.y = __uint_as_float(v[j + 1]) * rs;
            o.z = __uint_as_float(v[j + 2]) * rs;
            o.w = __uint_as_float(v[j + 3]) * rs;
            *reinterpret_cast<float4*>(buf + sw128_offset(lane, j >> 2)) = o;
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int x = static_cast<int>(col), yy = static_cast<int>(m0 + quarter * 32);
            if (p.accumulate) tma_reduce_add_3d(&tma_c, smem_u32(buf), x, yy, b);
            else tma_store_3d(&tma_c, smem_u32(buf), x, yy, b);
            tma_store_commit();
          }
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t v[32];
          tmem_ld32(t_row + c, v);
          tmem_ld_wait();
          const int64_t col = n0 + c;
          if (row_ok && col < p.N) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              if (col + j + 4 <= p.N) {
                float4 o;
                o.x = __uint_as_float(v[j]) * rs;
                o.y = __uint_as_float(v[j + 1]) * rs;
                o.z = __uint_as_float(v[j + 2]) * rs;
                o.w = __uint_as_float(v[j + 3]) * rs;
                const float4 cv = *reinterpret_cast<const float4*>(cin_row + col + j);
                o.x += p.beta * cv.x; o.y += p.beta * cv.y; o.z += p.beta * cv.z; o.w += p.beta * cv.w;
                *reinterpret_cast<float4*>(crow + col + j) = o;
              } else {
                for (int e = 0; e < 4 && col + j + e < p.N; ++e) {
                  crow[col + j + e] = __uint_as_float(v[j + e]) * rs + p.beta * cin_row[col + j + e];
                }
              }
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(acc));
      acc_phase[acc] ^= 1u;
      acc ^= 1;
    }
    if ((sizeof(OutT) == 2 || !HAS_CIN) && lane == 0) tma_store_wait0();   // staging buffers stay valid until the stores ran
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int BN, int STAGES, bool A_MN, bool B_MN, typename OutT, bool HAS_CIN, bool SWIGLU = false>
static int launch_gemm(const CUtensorMap& ta, const GemmBMaps& tb, const CUtensorMap& tc, void* c, const void* cin,
                       const GemmParams& p, cudaStream_t stream) {
  using S = GemmSmem<BN, STAGES>;
  auto kern = gemm_kernel<BN, STAGES, A_MN, B_MN, OutT, HAS_CIN, SWIGLU>;
  constexpr int smem_bytes = S::TOTAL + 1024;
  static bool configured = false;  // per instantiation; attribute is per function, device-independent here
  if (!configured) {
    TTCD_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    configured = true;
  }
  const int64_t total = p.tiles_m * p.tiles_n * p.batch;
  const int grid = static_cast<int>(total < sm_count() ? total : sm_count());
  launch_after(total <= sm_count(), kern, grid, gemm_threads(BN, SWIGLU), smem_bytes, stream, ta, tb, tc, static_cast<OutT*>(c), static_cast<const OutT*>(cin), p);
  return static_cast<int>(cudaGetLastError());
}

template <int BN, int STAGES, bool A_MN, bool B_MN>
static int dispatch_out(const CUtensorMap& ta, const GemmBMaps& tb, const CUtensorMap& tc, void* c, const void* cin,
                        const GemmParams& p, int out_fp32, cudaStream_t stream) {
  const bool has_cin = cin != nullptr && p.beta != 0.f && !p.accumulate;
  if (out_fp32) {
    return has_cin ? launch_gemm<BN, STAGES, A_MN, B_MN, float, true>(ta, tb, tc, c, cin, p, stream)
                   : launch_gemm<BN, STAGES, A_MN, B_MN, float, false>(ta, tb, tc, c, cin, p, stream);
  }
  return has_cin ? launch_gemm<BN, STAGES, A_MN, B_MN, bf16, true>(ta, tb, tc, c, cin, p, stream)
                 : launch_gemm<BN, STAGES, A_MN, B_MN, bf16, false>(ta, tb, tc, c, cin, p, stream);
}

template <int BN, int STAGES>
static int dispatch_major(const CUtensorMap& ta, const GemmBMaps& tb, const CUtensorMap& tc, void* c, const void* cin,
                          const GemmParams& p, int a_mn, int b_mn, int out_fp32, cudaStream_t stream) {
  if (!a_mn && !b_mn) return dispatch_out<BN, STAGES, false, false>(ta, tb, tc, c, cin, p, out_fp32, stream);
  if (!a_mn && b_mn) return dispatch_out<BN, STAGES, false, true>(ta, tb, tc, c, cin, p, out_fp32, stream);
  if (a_mn && !b_mn) return dispatch_out<BN, STAGES, true, false>(ta, tb, tc, c, cin, p, out_fp32, stream);
  return dispatch_out<BN, STAGES, true, true>(ta, tb, tc, c, cin, p, out_fp32, stream);
}

// Width of a tile.  256 columns are the cheapest per flop (operand traffic), but a grid of tiles runs in whole waves of the SMs,
// and where the last wave is nearly empty, or the only one has few tiles, narrower tiles finish earlier.  Time of a launch in
// units of one wave of 256-wide tiles, fitted to 230 shapes of the shipped models (M 300 .. 131072, N 1024 .. 128256, K 1024 ..
// 128256): waves at 256; 0.56 waves + 0.07 at 128; 0.42 waves + 0.12 at 64.  us at 256 | 128 | 64:
//   one wave, few tiles: 300 x 1024 x 3072: 25.6 | 19.5 | 17.4; 448 x 2048 x 8192: 57 | 38 | 31; 2048 x 1024 x 32000: 178 | 118 | 168
//   a second wave that is nearly empty: 6002 x 1024 x 3072: 46 | 42 | 56; 6144 x 1024 x 22646: 259 | 228 | 345
//   full waves: 3832 x 1024 x 3072: 28 | 32 | 41; 32768 x 1024 x 2816: 131 | 147 | 207
static double gemm_tile_cost(int bn, int64_t M, int64_t N, int64_t batch) {
  const int64_t rows = (M + GEMM_BM - 1) / GEMM_BM * batch, sms = sm_count();
  const double waves = static_cast<double>((rows * ((N + bn - 1) / bn) + sms - 1) / sms);
  return bn == 256 ? waves : bn == 128 ? 0.56 * waves + 0.07 : 0.42 * waves + 0.12;
}
static int gemm_tile_n(int64_t M, int64_t N, int64_t batch) {
  int best = 128;
  double cost = gemm_tile_cost(128, M, N, batch);
  const double narrow = gemm_tile_cost(64, M, N, batch);
  if (narrow < cost) { best = 64; cost = narrow; }
  return N >= 256 && gemm_tile_cost(256, M, N, batch) <= 1.06 * cost ? 256 : best;      // (5003 x 2048 x 2048, 3 | 2.87: 44 for 46 alone, no gain between others)
}

// The widest tile, bn columns at most, whose rows of B come from one matrix each (n3 may be 0) and whose box fits in it; 0: none.
static int gemm_piece_width(int bn, int64_t n1, int64_t n2, int64_t n3) {
  int64_t least = n1 < n2 ? n1 : n2;
  if (n3 > 0 && n3 < least) least = n3;
  for (; bn >= 64; bn /= 2)
    if (n1 % bn == 0 && (n3 == 0 || n2 % bn == 0) && least >= bn) return bn;
  return 0;
}

}  // namespace ttcd

TTCD_DEFINE_STATUS_READER(gemm)

// a: [batch][M][K] (a_mn = 0, row stride lda) or [batch][K][M] (a_mn = 1).  b likewise with N.
// c / c_in: [batch][M][N], row stride ldc, bf16 or fp32 (out_fp32).  Strides in elements.
// c_in may alias c.  row_scale: optional bf16 [batch*M].
int ttcd::gemm_run(const GemmCall& g, cudaStream_t stream) {
  const int64_t M = g.M, N = g.N, K = g.K, batch = g.batch;
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return TTCD_ERR_ARG;
  if (g.lse_part != nullptr && (g.out_fp32 || (reinterpret_cast<uintptr_t>(g.lse_part) & 7u))) return TTCD_ERR_ARG;
  const int elem_c = g.out_fp32 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(g.c) & 15u) || (g.ldc * elem_c) % 16 != 0 || (g.stride_c * elem_c) % 16 != 0)
    return TTCD_ERR_ARG;
  if (g.c_in != nullptr && (reinterpret_cast<uintptr_t>(g.c_in) & 15u)) return TTCD_ERR_ARG;
  // every TMA box must fit inside its tensor: the caller pads tiny problems up to these minima
  if (M < GEMM_BM || N < 128 || K < GEMM_BK) return TTCD_ERR_ARG;
  const bool pieces = g.swiglu || g.n1 != 0;
  if (pieces && (g.b_mn || batch != 1 || g.lse_part != nullptr || g.b2 == nullptr)) return TTCD_ERR_ARG;
  if (g.swiglu && (g.a_mn || g.out_fp32 || g.c_in != nullptr || g.n1 != 0)) return TTCD_ERR_ARG;
  if (g.round_first && (g.out_fp32 || g.c_in == nullptr || g.beta != 1.f)) return TTCD_ERR_ARG;
  const int64_t n3 = N - g.n1 - g.n2;
  if (g.n1 != 0 && (g.n1 < 0 || g.n2 <= 0 || n3 < 0 || (n3 > 0 && g.b3 == nullptr))) return TTCD_ERR_ARG;
  // the rows of B per tile (with SwiGLU gate and up; the pairs of lse_part are per 256 or 128 columns, as the caller sized it)
  int BN = g.lse_part != nullptr ? (N >= 256 ? 256 : 128) : gemm_tile_n(M, g.swiglu ? 2 * N : N, batch);
  if (g.swiglu && BN < 128) BN = 128;              // (a box of C is 64 columns wide)
  if (g.n1 != 0) {                                 // a tile's rows of B come from one matrix, and its box fits in it
    BN = gemm_piece_width(BN, g.n1, g.n2, n3);
    if (BN == 0) return TTCD_ERR_ARG;
  }
  CUtensorMap ta;
  GemmBMaps tb;
  int rc;
  const int a_bcast = (batch > 1 && g.stride_a == 0) ? 1 : 0;
  const int b_bcast = (batch > 1 && g.stride_b == 0) ? 1 : 0;
  const int64_t batch_a = a_bcast ? 1 : batch, batch_b = b_bcast ? 1 : batch;
  if (!g.a_mn) rc = make_tmap_bf16_3d(&ta, g.a, K, M, batch_a, g.lda, g.stride_a, 64, GEMM_BM);
  else         rc = make_tmap_bf16_3d(&ta, g.a, M, K, batch_a, g.lda, g.stride_a, 64, GEMM_BK);
  if (rc != TTCD_OK) return rc;
  if (g.b_mn) rc = make_tmap_bf16_3d(&tb.m[0], g.b, N, K, batch_b, g.ldb, g.stride_b, 64, GEMM_BK);
  else        rc = make_tmap_bf16_3d(&tb.m[0], g.b, K, g.n1 != 0 ? g.n1 : N, batch_b, g.ldb, g.stride_b, 64, g.swiglu ? BN / 2 : BN);
  if (rc != TTCD_OK) return rc;
  tb.m[1] = tb.m[2] = tb.m[0];
  if (pieces) {
    rc = make_tmap_bf16_3d(&tb.m[1], g.b2, K, g.swiglu ? N : g.n2, 1, g.ldb, 0, 64, g.swiglu ? BN / 2 : BN);
    if (rc == TTCD_OK && g.n1 != 0 && n3 > 0) rc = make_tmap_bf16_3d(&tb.m[2], g.b3, K, n3, 1, g.ldb, 0, 64, BN);
    if (rc != TTCD_OK) return rc;
  }
  const int CN = g.swiglu ? BN / 2 : BN;
  GemmParams p;
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.ldc = g.ldc; p.stride_c = g.stride_c;
  p.tiles_m = (M + GEMM_BM - 1) / GEMM_BM;
  p.tiles_n = (N + CN - 1) / CN;
  p.alpha = g.alpha; p.beta = g.beta;
  p.row_scale = static_cast<const bf16*>(g.row_scale);
  p.a_bcast = a_bcast; p.b_bcast = b_bcast;
  p.seg1 = g.n1 != 0 ? g.n1 : INT64_MAX;
  p.seg2 = g.n1 != 0 && n3 > 0 ? g.n1 + g.n2 : INT64_MAX;
  p.round_first = g.round_first;
  // the operand panel that is re-streamed once per step of the outer tile loop should be the smaller one (it then
  // lives in the 126 MB L2): walk M fastest when the B panel (N x K) is the larger
  p.m_fastest = (g.swiglu ? 2 * N : N) > M ? 1 : 0;
  p.lse_part = reinterpret_cast<float2*>(g.lse_part);
  // adding to C where it stands needs no read of C; not when batch entries share C (their order would not be fixed)
  p.accumulate = g.out_fp32 && g.c_in == g.c && g.beta == 1.f && (batch == 1 || g.stride_c != 0) ? 1 : 0;
  CUtensorMap tc;
  rc = g.out_fp32 ? make_tmap_f32_3d(&tc, g.c, N, M, batch, g.ldc, g.stride_c, 32, 32)
                  : make_tmap_bf16_3d(&tc, g.c, N, M, batch, g.ldc, g.stride_c, 64, 32);
  if (rc != TTCD_OK) return rc;
  if (g.swiglu) {
    if (BN == 256) return launch_gemm<256, 4, false, false, bf16, false, true>(ta, tb, tc, g.c, nullptr, p, stream);
    return launch_gemm<128, 6, false, false, bf16, false, true>(ta, tb, tc, g.c, nullptr, p, stream);
  }
  if (BN == 256) return dispatch_major<256, 4>(ta, tb, tc, g.c, g.c_in, p, g.a_mn, g.b_mn, g.out_fp32, stream);
  if (BN == 64) return dispatch_major<64, 8>(ta, tb, tc, g.c, g.c_in, p, g.a_mn, g.b_mn, g.out_fp32, stream);
  return dispatch_major<128, 6>(ta, tb, tc, g.c, g.c_in, p, g.a_mn, g.b_mn, g.out_fp32, stream);
}

// Weights of 960 + 320 + 320 columns leave no wider tile than 64, which costs 0.42 of a 256-wide one for a quarter of the columns; three
// copies of a few MB take ~12 us, a unit of the cost ~6.7 ns of K.  us apart | copied, then one product:
//   960 + 320 + 320, K 960: 4000 rows: 26.7 | 31.8, 8000: 39.7 | 39.9, 16000: 67.6 | 58.4, 65536: 240 | 171
//   1024 + 192 + 192, K 1024: 8000 rows: 37.9 | 42.0, 16000: 63.6 | 60.4;  576 + 192 + 192, K 576: 16000: 32.8 | 40.0, 65536: 102 | 83
// 128-wide tiles are not worth the copies (2048 + 128 + 128, K 2048, 65536 rows: 453 | 462).
bool ttcd::gemm_pieces_slow(int64_t M, int64_t K, int64_t n1, int64_t n2, int64_t n3) {
  const int64_t N = n1 + n2 + n3;
  const int want = gemm_tile_n(M, N, 1);
  if (want == 64 || gemm_piece_width(want, n1, n2, n3) != 64) return false;
  return (gemm_tile_cost(64, M, N, 1) - gemm_tile_cost(want, M, N, 1)) * static_cast<double>(K) > 1800.0;
}

TTCD_EXPORT int ttcd_gemm_bf16(const void* a, const void* b, void* c, const void* c_in, const void* row_scale,
                               long long M, long long N, long long K, long long batch, long long lda,
                               long long ldb, long long ldc, long long stride_a, long long stride_b,
                               long long stride_c, int a_mn, int b_mn, int out_fp32, float alpha, float beta,
                               void* stream_ptr) {
  ttcd::GemmCall g;
  g.a = a; g.b = b; g.c = c; g.c_in = c_in; g.row_scale = row_scale;
  g.M = M; g.N = N; g.K = K; g.batch = batch; g.lda = lda; g.ldb = ldb; g.ldc = ldc;
  g.stride_a = stride_a; g.stride_b = stride_b; g.stride_c = stride_c;
  g.a_mn = a_mn; g.b_mn = b_mn; g.out_fp32 = out_fp32; g.alpha = alpha; g.beta = beta;
  return ttcd::gemm_run(g, static_cast<cudaStream_t>(stream_ptr));
}

// Same GEMM (bf16 output) that also leaves, per output row and column tile, the pair (max, sum of exp(x - max)) of the
// row's values in that tile, taken on the bf16-rounded outputs: lse_part is fp32 [batch*M][tiles_n][2] with
// tiles_n = ceil(N / 256) (N >= 256) or ceil(N / 128).  A consumer merges the tiles_n pairs of a row into its
// log-sum-exp without reading the row (the cross-entropy row kernel does).
TTCD_EXPORT int ttcd_gemm_bf16_lse(const void* a, const void* b, void* c, long long M, long long N, long long K,
                                   long long lda, long long ldb, long long ldc, int a_mn, int b_mn, float alpha,
                                   float* lse_part, void* stream_ptr) {
  if (lse_part == nullptr) return TTCD_ERR_ARG;
  ttcd::GemmCall g;
  g.a = a; g.b = b; g.c = c; g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.stride_c = M * ldc;
  g.a_mn = a_mn; g.b_mn = b_mn; g.alpha = alpha; g.lse_part = lse_part;
  return ttcd::gemm_run(g, static_cast<cudaStream_t>(stream_ptr));
}

// Products of inference (K-major operands, bf16 [M, K] times rows of B): up to three matrices side by side (b [n1, K], b2 [n2, K],
// b3 the rest; n1 = 0: b alone), res (may be null, [M, N] like c) added to the rounded product, swiglu of b (gate) and b2 (up).
TTCD_EXPORT int ttcd_gemm_pieces(const void* a, const void* b, const void* b2, const void* b3, void* c, const void* res, long long M,
                                 long long N, long long K, long long lda, long long ldb, long long ldc, long long n1, long long n2,
                                 int swiglu, void* stream_ptr) {
  ttcd::GemmCall g;
  g.a = a; g.b = b; g.b2 = b2; g.b3 = b3; g.c = c; g.c_in = res; g.beta = res != nullptr ? 1.f : 0.f; g.round_first = res != nullptr;
  g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb; g.ldc = ldc; g.stride_c = M * ldc; g.n1 = n1; g.n2 = n2; g.swiglu = swiglu;
  return ttcd::gemm_run(g, static_cast<cudaStream_t>(stream_ptr));
}
