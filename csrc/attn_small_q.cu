// Attention for a few query rows over a long key/value cache (sm_100a): the decode step (one row) and short
// continuations (up to 127 rows), where a 128-row tensor-core tile would be almost empty and the work is one
// pass over the cached keys and values.
//
//   pass 1 (attn_small_q_partial): grid (key splits, kv heads, batch).  A CTA stages its <= 256 keys and values in
//           shared memory with 16-byte loads (rows padded by 16 bytes: conflict-free row-per-lane reads), then each
//           warp takes (query row, head of the GQA group) pairs: lanes own keys for Q.K (fp32, the query in shared
//           memory), the warp reduces max / sum, lanes own head-dim slices for P.V.  Writes the partial output and
//           its (max, sum) per split.
//   pass 2 (attn_small_q_merge): one CTA per (batch, head, row) folds the splits with the log-sum-exp identity.
//
// Up to 8 (row, head) pairs per key/value head (a decode step of grouped-query attention) take attn_decode_partial
// instead of pass 1: bound by reading the cache once, so keys and values go from global memory straight to registers.
//
// Causal mask with bottom-right alignment (query row r sits at key position Tk - Tq + r) and an optional sliding
// window, as flash_attn_func(causal=True, window_size=(W-1, 0)) applies them on the cached decode path of the
// reference (fla/layers/attn.py:215-226, 271-282).  Forward only.
#include "common.cuh"

namespace ttcd {

constexpr int SQ_KEYS = 256;       // keys per split
constexpr int SQ_WARPS = 8;

template <int D>
struct SmallQSmem {
  static constexpr int ROW_BYTES = D * 2 + 16;                    // padded K / V row
  static constexpr int K_OFF = 0;
  static constexpr int V_OFF = K_OFF + SQ_KEYS * ROW_BYTES;
  static constexpr int Q_OFF = V_OFF + SQ_KEYS * ROW_BYTES;       // SQ_WARPS query rows, fp32
  static constexpr int P_OFF = Q_OFF + SQ_WARPS * D * 4;          // SQ_WARPS x SQ_KEYS probabilities, fp32
  static constexpr int TOTAL = P_OFF + SQ_WARPS * SQ_KEYS * 4;
};

struct SmallQParams {
  const bf16* q; const bf16* k; const bf16* v;
  float* part_o;        // [B, H, Tq, splits, D]
  float* part_ml;       // [B, H, Tq, splits, 2]  (max in log2 units, sum)
  bf16* out;            // [B, Tq, H, D]
  int* turns;           // optional [B * HK], zero: CTAs that have finished; the last one of a head merges the splits
  const int* kv_len;    // optional device word: the number of valid keys (<= Tk); read at launch time
  int B, Tq, Tk, H, HK, splits, window;
  int64_t ldq, ldk, ldv, sq, sk, sv;
  float scale_log2;
};

template <int D>
__global__ void __launch_bounds__(SQ_WARPS * 32) attn_small_q_partial_kernel(const SmallQParams p) {
  using S = SmallQSmem<D>;
  extern __shared__ __align__(16) uint8_t smem[];
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = p.H / p.HK;
  const int key0 = split * SQ_KEYS;
  // a cache with a device-side fill count: splits past the count stage nothing and report an empty partial
  const int Tk = p.kv_len != nullptr ? min(max(*p.kv_len, p.Tq), p.Tk) : p.Tk;
  const int nkeys = min(SQ_KEYS, Tk - key0);
  constexpr int VPR = D / 8;                                     // 16-byte vectors per row
  // ---- stage K and V rows of this split
  for (int i = threadIdx.x; i < nkeys * VPR; i += blockDim.x) {
    const int r = i / VPR, c = i % VPR;
    const int64_t krow = static_cast<int64_t>(b) * p.sk + static_cast<int64_t>(key0 + r) * p.ldk + kvh * D + c * 8;
    const int64_t vrow = static_cast<int64_t>(b) * p.sv + static_cast<int64_t>(key0 + r) * p.ldv + kvh * D + c * 8;
    *reinterpret_cast<uint4*>(smem + S::K_OFF + r * S::ROW_BYTES + c * 16) = *reinterpret_cast<const uint4*>(p.k + krow);
    *reinterpret_cast<uint4*>(smem + S::V_OFF + r * S::ROW_BYTES + c * 16) = *reinterpret_cast<const uint4*>(p.v + vrow);
  }
  __syncthreads();
  float* qs = reinterpret_cast<float*>(smem + S::Q_OFF) + warp * D;
  float* ps = reinterpret_cast<float*>(smem + S::P_OFF) + warp * SQ_KEYS;
  const int npairs = p.Tq * G;
  for (int pair = warp; pair < npairs; pair += SQ_WARPS) {
    const int row = pair / G, h = kvh * G + pair % G;
    const int qpos = Tk - p.Tq + row;
    const int lo_excl = p.window > 0 ? qpos - p.window : -1;
    // the query row -> shared memory as fp32
    const bf16* qrow = p.q + static_cast<int64_t>(b) * p.sq + static_cast<int64_t>(row) * p.ldq + h * D;
    for (int d = lane; d < D; d += 32) qs[d] = __bfloat162float(qrow[d]);
    __syncwarp();
    // ---- scores: lane owns keys lane, lane + 32, ...
    float sc[SQ_KEYS / 32];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < SQ_KEYS / 32; ++j) {
      const int r = lane + 32 * j, key = key0 + r;
      float acc = 0.f;
      if (r < nkeys && key <= qpos && key > lo_excl) {
        const uint8_t* krow = smem + S::K_OFF + r * S::ROW_BYTES;
#pragma unroll 4
        for (int c = 0; c < VPR; ++c) {
          const uint4 raw = *reinterpret_cast<const uint4*>(krow + c * 16);
          const float4 qa = *reinterpret_cast<const float4*>(qs + c * 8), qb = *reinterpret_cast<const float4*>(qs + c * 8 + 4);
          const float2 k0 = unpack_bf16(raw.x), k1 = unpack_bf16(raw.y), k2 = unpack_bf16(raw.z), k3 = unpack_bf16(raw.w);
          acc = fmaf(k0.x, qa.x, acc); acc = fmaf(k0.y, qa.y, acc);
          acc = fmaf(k1.x, qa.z, acc); acc = fmaf(k1.y, qa.w, acc);
          acc = fmaf(k2.x, qb.x, acc); acc = fmaf(k2.y, qb.y, acc);
          acc = fmaf(k3.x, qb.z, acc); acc = fmaf(k3.y, qb.w, acc);
        }
        acc *= p.scale_log2;
      } else {
        acc = -INFINITY;
      }
      sc[j] = acc;
      mx = fmaxf(mx, acc);
    }
    mx = warp_max(mx);
    const float m_use = mx == -INFINITY ? 0.f : mx;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < SQ_KEYS / 32; ++j) {
      const float e = exp2f(sc[j] - m_use);          // exp2(-inf) = 0 for masked keys
      ps[lane + 32 * j] = e;
      sum += e;
    }
    sum = warp_sum(sum);
    __syncwarp();
    // ---- output: lane owns D / 32 consecutive head-dim elements
    constexpr int DPL = D / 32;
    float o[DPL];
#pragma unroll
    for (int e = 0; e < DPL; ++e) o[e] = 0.f;
    for (int r = 0; r < nkeys; ++r) {
      const float pr = ps[r];
      const bf16* vrow = reinterpret_cast<const bf16*>(smem + S::V_OFF + r * S::ROW_BYTES) + lane * DPL;
      if (DPL == 4) {
        const uint2 raw = *reinterpret_cast<const uint2*>(vrow);
        const float2 a = unpack_bf16(raw.x), c = unpack_bf16(raw.y);
        o[0] = fmaf(pr, a.x, o[0]); o[1] = fmaf(pr, a.y, o[1]);
        o[DPL - 2] = fmaf(pr, c.x, o[DPL - 2]); o[DPL - 1] = fmaf(pr, c.y, o[DPL - 1]);
      } else {
        const float2 a = unpack_bf16(*reinterpret_cast<const uint32_t*>(vrow));
        o[0] = fmaf(pr, a.x, o[0]); o[1] = fmaf(pr, a.y, o[1]);
      }
    }
    const int64_t pidx = ((static_cast<int64_t>(b) * p.H + h) * p.Tq + row) * p.splits + split;
#pragma unroll
    for (int e = 0; e < DPL; ++e) p.part_o[pidx * D + lane * DPL + e] = o[e];
    if (lane == 0) {
      p.part_ml[pidx * 2] = mx;
      p.part_ml[pidx * 2 + 1] = sum;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------------------------------------------
// At most R (query row, head of the group) pairs per key/value head.  D / 8 lanes hold a cached row (16 bytes each),
// so a warp-wide load brings KPW = 32 / (D / 8) keys; a warp takes U such loads of K and of V at a time, all issued
// before the first use.  A lane forms the products of its 8 dims for U keys x R pairs, a transposing reduction over
// the lanes of a key leaves every lane with NV = U R / (D / 8) whole scores (so that each exponential is computed
// once), and the probabilities travel back by shuffles for the fp32 P V.  Running max per pair, moved only when it
// grows by 2^8.  No shared memory until the warps of a CTA are merged.
// The fill count decides the split borders: a captured launch cuts what is filled into as many ranges as it has CTAs per head
// (whole turns each; the last ones are empty while little is filled).  With up to two pairs a CTA has at most 124 registers
// per thread and two fit an SM; four and eight pairs take 182 to 232, one fits.
// Bound by the cache's bytes: 8 x 8192 keys, 16/8 heads, D 128 (268 MB): 46 us, 0.9 of the copy rate.  1 x 8192 (33.6 MB):
// 11 us; the staging kernel above took 40.8 us (135 KB of shared memory, so one CTA per SM that first loads and then
// computes, 1.7 waves).
constexpr int DEC_WARPS = 8;

template <int D, int R>
struct DecodeCfg {
  static constexpr int LPR = D / 8;                 // lanes per cached row
  static constexpr int KPW = 32 / LPR;              // keys per warp-wide load
  static constexpr int U = R <= 4 ? 8 : 4;          // loads in flight (of K and of V each)
  static constexpr int KEYS = KPW * U;              // keys per warp and turn
  static constexpr int N = U * R;                   // scores per lane group and turn
  static constexpr int NV = N >= LPR ? N / LPR : 1; // ... of which a lane ends up with
  static constexpr int DUP = N >= LPR ? 1 : LPR / N;// lanes that hold the same score
};

template <int D, int R>
__global__ void __launch_bounds__(DEC_WARPS * 32, R <= 2 ? 2 : 1) attn_decode_partial_kernel(const SmallQParams p) {
  using C = DecodeCfg<D, R>;
  constexpr int LPR = C::LPR, KPW = C::KPW, U = C::U, NV = C::NV, DUP = C::DUP;
  static_assert(NV <= R && (R & (R - 1)) == 0, "a lane's scores belong to different pairs");
  __shared__ float s_m[DEC_WARPS * KPW][R], s_l[DEC_WARPS * KPW][R];
  __shared__ __align__(16) float s_o[DEC_WARPS][R][D];
  pdl_wait();
  pdl_launch_dependents();
  const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = lane / LPR, l = lane % LPR;       // key of a load, lane of the key
  const int G = p.H / p.HK, pairs = p.Tq * G;
  const int Tk = p.kv_len != nullptr ? min(max(*p.kv_len, p.Tq), p.Tk) : p.Tk;
  // keys [first, Tk) are seen by some row; a split takes a multiple of the CTA's keys per turn
  const int first = p.window > 0 ? max(0, Tk - p.Tq - p.window + 1) : 0;
  constexpr int TURN = DEC_WARPS * C::KEYS;
  const int per = ((Tk - first + p.splits - 1) / p.splits + TURN - 1) / TURN * TURN;
  const int lo = first + split * per, hi = min(Tk, lo + per);
  // this lane's 8 dims of every query pair (pairs beyond the real ones: zero)
  float2 q[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    uint4 raw = make_uint4(0u, 0u, 0u, 0u);
    if (r < pairs)
      raw = *reinterpret_cast<const uint4*>(p.q + static_cast<int64_t>(b) * p.sq + static_cast<int64_t>(r / G) * p.ldq +
                                            (kvh * G + r % G) * D + l * 8);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      q[r][i] = unpack_bf16(w[i]);
    }
  }
  const bf16* kbase = p.k + static_cast<int64_t>(b) * p.sk + kvh * D + l * 8;
  const bf16* vbase = p.v + static_cast<int64_t>(b) * p.sv + kvh * D + l * 8;

  float2 o[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < 4; ++i) o[r][i] = make_float2(0.f, 0.f);
  // the scores this lane ends up with: n = own0 + j, pair n % R, key n / R
  const int own0 = (l / DUP) * NV;
  float m_ref[NV], l_sum[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) { m_ref[j] = -INFINITY; l_sum[j] = 0.f; }

  for (int t0 = lo + warp * C::KEYS; t0 < hi; t0 += TURN) {
    uint4 kr[U], vr[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {                   // rows past the end re-read the last one (masked below)
      const int64_t key = min(t0 + u * KPW + grp, Tk - 1);
      kr[u] = *reinterpret_cast<const uint4*>(kbase + key * p.ldk);
      vr[u] = *reinterpret_cast<const uint4*>(vbase + key * p.ldv);
    }
    float sc[C::N];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float2 k0 = unpack_bf16(kr[u].x), k1 = unpack_bf16(kr[u].y), k2 = unpack_bf16(kr[u].z), k3 = unpack_bf16(kr[u].w);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float2 a = __fmul2_rn(q[r][0], k0);
        a = __ffma2_rn(q[r][1], k1, a);
        a = __ffma2_rn(q[r][2], k2, a);
        a = __ffma2_rn(q[r][3], k3, a);
        sc[u * R + r] = a.x + a.y;
      }
    }
    // transposing reduction over the lanes of a key: halve the scores while there are several, then plain sums
#pragma unroll
    for (int d = LPR / 2, n = C::N; d > 0; d >>= 1) {
      const bool up = (l & d) != 0;
      if (n > 1) {
        n >>= 1;
#pragma unroll
        for (int i = 0; i < C::N / 2; ++i)
          if (i < n) {
            const float send = up ? sc[i] : sc[n + i], keep = up ? sc[n + i] : sc[i];
            sc[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
          }
      } else {
        sc[0] += __shfl_xor_sync(0xffffffffu, sc[0], d);
      }
    }
    float pr[NV];
    bool need = false;
    float m_new[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int n = own0 + j, r = n % R, key = t0 + (n / R) * KPW + grp;
      const int qpos = Tk - p.Tq + r / G;
      const bool vis = key < hi && key <= qpos && (p.window <= 0 || key > qpos - p.window);
      pr[j] = vis ? sc[j] * p.scale_log2 : -INFINITY;
      float m = pr[j];
#pragma unroll
      for (int d = R / NV * DUP; d < LPR; d <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));   // over the keys
      m_new[j] = fmaxf(m, m_ref[j]);
      need = need || m_new[j] > m_ref[j] + 8.f || (m_ref[j] == -INFINITY && m_new[j] > -INFINITY);
    }
    if (__any_sync(0xffffffffu, need)) {
      float f[NV];
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        f[j] = m_ref[j] == -INFINITY ? 0.f : exp2f(m_ref[j] - m_new[j]);
        l_sum[j] *= f[j];
        m_ref[j] = m_new[j];
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float fr = __shfl_sync(0xffffffffu, f[r % NV], r / NV * DUP, LPR);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[r][i] = make_float2(o[r][i].x * fr, o[r][i].y * fr);
      }
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      pr[j] = pr[j] == -INFINITY ? 0.f : exp2f(pr[j] - m_ref[j]);
      l_sum[j] += pr[j];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float2 v0 = unpack_bf16(vr[u].x), v1 = unpack_bf16(vr[u].y), v2 = unpack_bf16(vr[u].z), v3 = unpack_bf16(vr[u].w);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int n = u * R + r;
        const float e = __shfl_sync(0xffffffffu, pr[n % NV], n / NV * DUP, LPR);
        const float2 e2 = make_float2(e, e);
        o[r][0] = __ffma2_rn(e2, v0, o[r][0]);
        o[r][1] = __ffma2_rn(e2, v1, o[r][1]);
        o[r][2] = __ffma2_rn(e2, v2, o[r][2]);
        o[r][3] = __ffma2_rn(e2, v3, o[r][3]);
      }
    }
  }
  // ---- merge the lane groups of all warps: row (warp, group) of s_m / s_l, then one common max per pair
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    float s = l_sum[j];
#pragma unroll
    for (int d = R / NV * DUP; d < LPR; d <<= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (l < R / NV * DUP && l % DUP == 0) {         // the lanes of the first key hold every pair once
      s_m[warp * KPW + grp][(own0 + j) % R] = m_ref[j];
      s_l[warp * KPW + grp][(own0 + j) % R] = s;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float M = -INFINITY;
#pragma unroll
    for (int i = 0; i < DEC_WARPS * KPW; ++i) M = fmaxf(M, s_m[i][r]);
    const float mine = s_m[warp * KPW + grp][r];
    const float f = mine == -INFINITY ? 0.f : exp2f(mine - M);
    float x[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) { x[2 * i] = o[r][i].x * f; x[2 * i + 1] = o[r][i].y * f; }
#pragma unroll
    for (int d = LPR; d < 32; d <<= 1)
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] += __shfl_xor_sync(0xffffffffu, x[i], d);
    if (grp == 0) {
      *reinterpret_cast<float4*>(&s_o[warp][r][l * 8]) = make_float4(x[0], x[1], x[2], x[3]);
      *reinterpret_cast<float4*>(&s_o[warp][r][l * 8 + 4]) = make_float4(x[4], x[5], x[6], x[7]);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < pairs * D; i += DEC_WARPS * 32) {
    const int r = i / D, d = i % D;
    float acc = 0.f;
#pragma unroll
    for (int w = 0; w < DEC_WARPS; ++w) acc += s_o[w][r][d];
    const int64_t pidx = ((static_cast<int64_t>(b) * p.H + kvh * G + r % G) * p.Tq + r / G) * p.splits + split;
    p.part_o[pidx * D + d] = acc;
    if (d == 0) {
      float M = -INFINITY, s = 0.f;
      for (int w = 0; w < DEC_WARPS * KPW; ++w) M = fmaxf(M, s_m[w][r]);
      for (int w = 0; w < DEC_WARPS * KPW; ++w) s += s_m[w][r] == -INFINITY ? 0.f : s_l[w][r] * exp2f(s_m[w][r] - M);
      p.part_ml[pidx * 2] = M;
      p.part_ml[pidx * 2 + 1] = s;
    }
  }
  if (p.turns == nullptr) return;
  // ---- the last CTA of this (sample, head) folds the splits, as the merge kernel below does (a launch less: 3 us)
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    int* turn = p.turns + b * p.HK + kvh;
    s_last = atomicAdd(turn, 1) == p.splits - 1;
    if (s_last) *turn = 0;                          // as the next call finds it
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  constexpr int DPL = D / 32, WPP = DEC_WARPS / R;  // warps per pair
  const int r = warp / WPP, sub = warp % WPP;
  float* l_parts = &s_l[0][0];
  if (r < pairs) {
    const int64_t item = (static_cast<int64_t>(b) * p.H + kvh * G + r % G) * p.Tq + r / G;
    const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + item * p.splits;
    float M = -INFINITY;
    for (int s = lane; s < p.splits; s += 32) M = fmaxf(M, __ldcg(&ml[s]).x);
    M = warp_max(M);
    float acc[DPL], lsum = 0.f;
#pragma unroll
    for (int e = 0; e < DPL; ++e) acc[e] = 0.f;
    constexpr int MB = 8;                           // splits in flight, also where fewer are left
    for (int s0 = sub; s0 < p.splits; s0 += MB * WPP) {
      float2 t[MB];
      float x[MB][DPL];
#pragma unroll
      for (int u = 0; u < MB; ++u) {
        const int s = s0 + u * WPP;
        t[u] = s < p.splits ? __ldcg(&ml[s]) : make_float2(-INFINITY, 0.f);
#pragma unroll
        for (int e = 0; e < DPL; ++e) x[u][e] = s < p.splits ? __ldcg(p.part_o + (item * p.splits + s) * D + lane * DPL + e) : 0.f;
      }
#pragma unroll
      for (int u = 0; u < MB; ++u) {
        const bool some = t[u].x != -INFINITY;      // (an empty split counts for nothing)
        const float w = some ? exp2f(t[u].x - M) : 0.f;
        lsum = fmaf(some ? t[u].y : 0.f, w, lsum);
#pragma unroll
        for (int e = 0; e < DPL; ++e) acc[e] = fmaf(some ? x[u][e] : 0.f, w, acc[e]);
      }
    }
#pragma unroll
    for (int e = 0; e < DPL; ++e) s_o[sub][r][lane * DPL + e] = acc[e];
    if (lane == 0) l_parts[warp] = lsum;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < pairs * D; i += DEC_WARPS * 32) {
    const int pr = i / D, d = i % D;
    float acc = 0.f, tot = 0.f;
#pragma unroll
    for (int w = 0; w < WPP; ++w) { acc += s_o[w][pr][d]; tot += l_parts[pr * WPP + w]; }
    p.out[((static_cast<int64_t>(b) * p.Tq + pr / G) * p.H + kvh * G + pr % G) * D + d] = __float2bfloat16(acc * (tot > 0.f ? 1.f / tot : 0.f));
  }
}

// out[b, row, h, :] = sum_s o_s 2^(m_s - M) / sum_s l_s 2^(m_s - M): one CTA per item, warps over the splits, a lane
// owns D / 32 consecutive dims.  (One warp walking all splits in order took 8.7 us for 16 items of 32 splits.)
constexpr int MERGE_WARPS = 4;
template <int D>
__global__ void __launch_bounds__(MERGE_WARPS * 32) attn_small_q_merge_kernel(const SmallQParams p) {
  pdl_wait();
  pdl_launch_dependents();
  const int splits = p.splits, Tq = p.Tq, H = p.H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t item = blockIdx.x;                  // (b, h, row)
  constexpr int DPL = D / 32;
  __shared__ float s_o[MERGE_WARPS][D], s_l[MERGE_WARPS];
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + item * splits;
  float M = -INFINITY;
  for (int s = lane; s < splits; s += 32) M = fmaxf(M, ml[s].x);
  M = warp_max(M);
  float o[DPL], l = 0.f;
#pragma unroll
  for (int e = 0; e < DPL; ++e) o[e] = 0.f;
#pragma unroll 4
  for (int s = warp; s < splits; s += MERGE_WARPS) {
    const float2 t = ml[s];
    const float* src = p.part_o + (item * splits + s) * D + lane * DPL;
    float x[DPL];
#pragma unroll
    for (int e = 0; e < DPL; ++e) x[e] = src[e];
    const bool some = t.x != -INFINITY;             // an empty split: its partial output counts for nothing
    const float w = some ? exp2f(t.x - M) : 0.f;
    l = fmaf(some ? t.y : 0.f, w, l);
#pragma unroll
    for (int e = 0; e < DPL; ++e) o[e] = fmaf(some ? x[e] : 0.f, w, o[e]);
  }
#pragma unroll
  for (int e = 0; e < DPL; ++e) s_o[warp][lane * DPL + e] = o[e];
  if (lane == 0) s_l[warp] = l;
  __syncthreads();
  if (threadIdx.x < D) {
    float acc = 0.f, tot = 0.f;
#pragma unroll
    for (int w = 0; w < MERGE_WARPS; ++w) { acc += s_o[w][threadIdx.x]; tot += s_l[w]; }
    const int row = static_cast<int>(item % Tq);
    const int64_t bh = item / Tq, b = bh / H, h = bh % H;
    p.out[((b * Tq + row) * H + h) * D + threadIdx.x] = __float2bfloat16(acc * (tot > 0.f ? 1.f / tot : 0.f));
  }
}

template <int D>
static int launch_merge(const SmallQParams& p, cudaStream_t stream) {
  const int64_t items = static_cast<int64_t>(p.B) * p.H * p.Tq;
  return launch_dependent(attn_small_q_merge_kernel<D>, dim3(static_cast<unsigned>(items)), dim3(MERGE_WARPS * 32), 0, stream, p);
}

template <int D>
static int launch_decode(const SmallQParams& p, cudaStream_t stream) {
  const int pairs = p.Tq * (p.H / p.HK);
  auto kern = pairs <= 1 ? attn_decode_partial_kernel<D, 1> : pairs <= 2 ? attn_decode_partial_kernel<D, 2>
              : pairs <= 4 ? attn_decode_partial_kernel<D, 4> : attn_decode_partial_kernel<D, 8>;
  const int rc = launch_dependent(kern, dim3(p.splits, p.HK, p.B), dim3(DEC_WARPS * 32), 0, stream, p);
  return rc != TTCD_OK || p.turns != nullptr ? rc : launch_merge<D>(p, stream);
}

template <int D>
static int launch_small_q(const SmallQParams& p, cudaStream_t stream) {
  using S = SmallQSmem<D>;
  auto k1 = attn_small_q_partial_kernel<D>;
  static bool configured = false;
  if (!configured) {
    TTCD_CUDA_CHECK(cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL));
    configured = true;
  }
  k1<<<dim3(p.splits, p.HK, p.B), SQ_WARPS * 32, S::TOTAL, stream>>>(p);
  TTCD_CUDA_CHECK(cudaGetLastError());
  return launch_merge<D>(p, stream);
}

}  // namespace ttcd

// q [B, Tq, *] (token stride ldq, batch stride sq, head h at column h*D), k / v [B, Tk, *] likewise with HK heads,
// 16-byte aligned rows; out contiguous [B, Tq, H, D] bf16.  part_o fp32 [B, H, Tq, splits, D] and part_ml fp32
// [B, H, Tq, splits, 2] are caller-provided scratch; splits must equal ceil(Tk / 256).  window <= 0: unlimited.
// kv_len (may be null): a device int holding how many of the Tk key rows are filled, read when the kernel runs, so
// that a captured launch follows a cache that grows between replays; the causal alignment then counts from it.
static int small_q_params(ttcd::SmallQParams& p, const void* q, const void* k, const void* v, void* out, float* part_o, float* part_ml,
                          int B, int Tq, int Tk, int H, int HK, int D, long long ldq, long long ldk, long long ldv,
                          long long sq, long long sk, long long sv, int window, float scale, int splits, const int* kv_len) {
  using namespace ttcd;
  if (B <= 0 || Tq <= 0 || Tq >= 128 || Tk < Tq || H <= 0 || HK <= 0 || H % HK != 0 || (D != 64 && D != 128))
    return TTCD_ERR_ARG;
  if (ldk % 8 != 0 || ldv % 8 != 0 || sk % 8 != 0 || sv % 8 != 0) return TTCD_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(k) & 15u) || (reinterpret_cast<uintptr_t>(v) & 15u)) return TTCD_ERR_ARG;
  p.q = static_cast<const bf16*>(q); p.k = static_cast<const bf16*>(k); p.v = static_cast<const bf16*>(v);
  p.out = static_cast<bf16*>(out); p.part_o = part_o; p.part_ml = part_ml; p.kv_len = kv_len; p.turns = nullptr;
  p.B = B; p.Tq = Tq; p.Tk = Tk; p.H = H; p.HK = HK; p.splits = splits; p.window = window;
  p.ldq = ldq; p.ldk = ldk; p.ldv = ldv; p.sq = sq; p.sk = sk; p.sv = sv;
  p.scale_log2 = scale * 1.4426950408889634f;
  return TTCD_OK;
}

TTCD_EXPORT int ttcd_attn_small_q(const void* q, const void* k, const void* v, void* out, float* part_o, float* part_ml,
                                  int B, int Tq, int Tk, int H, int HK, int D, long long ldq, long long ldk, long long ldv,
                                  long long sq, long long sk, long long sv, int window, float scale, int splits,
                                  const int* kv_len, void* stream_ptr) {
  using namespace ttcd;
  if (splits != (Tk + SQ_KEYS - 1) / SQ_KEYS) return TTCD_ERR_ARG;
  SmallQParams p;
  const int rc = small_q_params(p, q, k, v, out, part_o, part_ml, B, Tq, Tk, H, HK, D, ldq, ldk, ldv, sq, sk, sv, window, scale,
                                splits, kv_len);
  if (rc != TTCD_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  return D == 128 ? launch_small_q<128>(p, stream)
                  : launch_small_q<64>(p, stream);
}

// The same call for at most 8 (query row, head of the group) pairs per key/value head: Tq * (H / HK) <= 8.  q rows are
// 16-byte aligned too; splits is any number from 1 to 65535 (the kernel cuts the filled keys into that many ranges).
// turns (may be null): int [B * HK], zero before the first call and left so by every call; calls that may overlap need their
// own.  With it the last CTA of a head merges the splits, without it a second launch does.
TTCD_EXPORT int ttcd_attn_decode(const void* q, const void* k, const void* v, void* out, float* part_o, float* part_ml,
                                 int B, int Tq, int Tk, int H, int HK, int D, long long ldq, long long ldk, long long ldv,
                                 long long sq, long long sk, long long sv, int window, float scale, int splits,
                                 int* turns, const int* kv_len, void* stream_ptr) {
  using namespace ttcd;
  if (splits < 1 || splits > 65535 || B > 65535 || HK > 65535) return TTCD_ERR_ARG;
  SmallQParams p;
  const int rc = small_q_params(p, q, k, v, out, part_o, part_ml, B, Tq, Tk, H, HK, D, ldq, ldk, ldv, sq, sk, sv, window, scale,
                                splits, kv_len);
  if (rc != TTCD_OK) return rc;
  if (Tq * (H / HK) > 8 || ldq % 8 != 0 || sq % 8 != 0 || (reinterpret_cast<uintptr_t>(q) & 15u)) return TTCD_ERR_ARG;
  p.turns = turns;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  return D == 128 ? launch_decode<128>(p, stream)
                  : launch_decode<64>(p, stream);
}
