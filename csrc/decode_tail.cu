// What surrounds the layers of a captured decode step: the choice of the next token with the move of the decoder's state, and
// the copy of a prompt's keys and values into the decoder's rings.  (The reference decodes eagerly through HF generate.)
#include "common.cuh"

namespace ttcd {

// The token that follows and the state of the next step, in one launch: per sample the index of the largest logit (the first
// one of equals; a NaN counts as largest, as torch.argmax has it), written to token[b] and out[b][cursor]; then cursor and
// position move on, and each ring's slot and fill count with them.  A token took ten library launches for it.
constexpr int PICK_RINGS = 4, PICK_SPLIT = 8, PICK_THREADS = 512;
struct PickParams {
  const bf16* logits; int64_t ld;                  // [B, V]
  int64_t* token; int64_t* out; int64_t out_ld;    // [B], [B, columns]
  int64_t *cursor, *pos, *positions;               // [1], [1], [B]
  int64_t* slot[PICK_RINGS]; int* kv_len[PICK_RINGS]; int64_t cap[PICK_RINGS];
  unsigned long long* best;                        // [B][PICK_SPLIT]
  int* turns;                                      // [1], zero before and after
  int B, V, columns, rings;
};

// larger key = larger logit; equal logits: the smaller index has the larger key
__device__ __forceinline__ unsigned long long pick_key(float v, int i) {
  uint32_t u = __float_as_uint(v);
  u = v != v ? 0xffffffffu : v == 0.f ? 0x80000000u : (u & 0x80000000u) ? ~u : u | 0x80000000u;
  return (static_cast<unsigned long long>(u) << 32) | (0xffffffffu - static_cast<uint32_t>(i));
}

__global__ void __launch_bounds__(PICK_THREADS) decode_pick_kernel(const PickParams p) {
  __shared__ unsigned long long s_best[PICK_THREADS / 32];
  __shared__ bool s_last;
  pdl_wait();
  pdl_launch_dependents();
  const int b = blockIdx.y, split = blockIdx.x;
  const int per = ((p.V + 7) / 8 + PICK_SPLIT - 1) / PICK_SPLIT * 8;
  const int lo = min(p.V, split * per), hi = min(p.V, lo + per);
  const bf16* row = p.logits + b * p.ld;
  unsigned long long best = 0;
  auto take = [&](unsigned long long k) { best = k > best ? k : best; };
  const int vec_hi = (reinterpret_cast<uintptr_t>(row) & 15u) == 0 ? lo + (hi - lo) / 8 * 8 : lo;
#pragma unroll 4
  for (int i = lo + threadIdx.x * 8; i < vec_hi; i += PICK_THREADS * 8) {
    float f[8];
    const uint4 v = *reinterpret_cast<const uint4*>(row + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) { const float2 t = unpack_bf16(w[e]); f[2 * e] = t.x; f[2 * e + 1] = t.y; }
#pragma unroll
    for (int e = 0; e < 8; ++e) take(pick_key(f[e], i + e));
  }
  for (int i = vec_hi + threadIdx.x; i < hi; i += PICK_THREADS) take(pick_key(__bfloat162float(row[i]), i));
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) take(__shfl_xor_sync(0xffffffffu, best, d));
  if ((threadIdx.x & 31) == 0) s_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < PICK_THREADS / 32; ++w) take(s_best[w]);
    __stcg(p.best + b * PICK_SPLIT + split, best);
    __threadfence();
    s_last = atomicAdd(p.turns, 1) == static_cast<int>(gridDim.x * gridDim.y) - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int64_t col = *p.cursor, pos = *p.pos + 1;
  __syncthreads();                                 // (read by all before they move)
  if (static_cast<int>(threadIdx.x) < p.B) {
    const int s = threadIdx.x;
    unsigned long long top = 0;
#pragma unroll
    for (int i = 0; i < PICK_SPLIT; ++i) { const unsigned long long k = __ldcg(p.best + s * PICK_SPLIT + i); top = k > top ? k : top; }
    const int64_t t = 0xffffffffu - static_cast<uint32_t>(top);
    p.token[s] = t;
    if (col >= 0 && col < p.columns) p.out[s * p.out_ld + col] = t;
    p.positions[s] = pos;
  }
  if (threadIdx.x == 0) {
    *p.turns = 0;
    *p.cursor = col + 1;
    *p.pos = pos;
    for (int i = 0; i < p.rings; ++i) {
      *p.slot[i] = pos % p.cap[i];
      *p.kv_len[i] = static_cast<int>(pos + 1 < p.cap[i] ? pos + 1 : p.cap[i]);
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// A prompt's keys and values into the rings of all layers, one launch: row i of n goes to ring row (start - n + i) % capacity.
// Bound by memory: 28 layers of 1 x 8192 rows x 2 KB (1.9 GB read and written) take what a copy takes; one indexed library copy
// per tensor took 26 us for each of 56.
constexpr int RING_LAYERS = 32, RING_THREADS = 256, RING_VECS = 4;
struct RingLayer { const bf16 *k, *v; bf16 *rk, *rv; int64_t sk_b, sk_r, sv_b, sv_r, ring_b; int rows, cap; };
struct RingParams {
  RingLayer layer[RING_LAYERS];
  int64_t start;
  int vecs;                                        // 16-byte vectors per row
};
static_assert(sizeof(RingParams) <= 4000, "kernel parameters");

__global__ void __launch_bounds__(RING_THREADS) ring_load_kernel(const __grid_constant__ RingParams p) {
  const RingLayer& L = p.layer[blockIdx.y >> 1];
  const bool is_v = blockIdx.y & 1;
  const int b = blockIdx.z;
  const int64_t sr = is_v ? L.sv_r : L.sk_r;
  const bf16* src = (is_v ? L.v + b * L.sv_b : L.k + b * L.sk_b);
  uint4* dst = reinterpret_cast<uint4*>((is_v ? L.rv : L.rk) + b * L.ring_b);
  const uint32_t total = static_cast<uint32_t>(L.rows) * p.vecs, vecs = p.vecs;
  const int first = static_cast<int>((p.start - L.rows) % L.cap);
  for (uint32_t i0 = blockIdx.x * (RING_THREADS * RING_VECS) + threadIdx.x; i0 < total; i0 += gridDim.x * (RING_THREADS * RING_VECS)) {
    uint4 x[RING_VECS];
#pragma unroll
    for (int u = 0; u < RING_VECS; ++u) {
      const uint32_t i = i0 + u * RING_THREADS;
      if (i < total) x[u] = *reinterpret_cast<const uint4*>(src + static_cast<int64_t>(i / vecs) * sr + i % vecs * 8);
    }
#pragma unroll
    for (int u = 0; u < RING_VECS; ++u) {
      const uint32_t i = i0 + u * RING_THREADS;
      if (i < total) {
        int row = first + static_cast<int>(i / vecs);
        if (row >= L.cap) row -= L.cap;
        dst[static_cast<int64_t>(row) * vecs + i % vecs] = x[u];
      }
    }
  }
}

}  // namespace ttcd

// logits [B, V] bf16 rows ld apart -> token [B], out [B, columns] at *cursor (nothing is written past the last column), then cursor,
// pos, positions [B] and the rings' (slot, kv_len, capacity; up to 4) move to the next token.  best: B * 8 int64 of scratch,
// turns: one int32, zero before the first call and left so.  B <= 512.
TTCD_EXPORT int ttcd_decode_pick(const void* logits, long long ld, int B, int V, long long* token, long long* out, long long out_ld,
                                 int columns, long long* cursor, long long* pos, long long* positions, long long** slots,
                                 int** kv_lens, const long long* caps, int rings, void* best, int* turns, void* stream_ptr) {
  using namespace ttcd;
  if (B < 1 || B > PICK_THREADS || V < 1 || rings < 0 || rings > PICK_RINGS) return TTCD_ERR_ARG;
  PickParams p;
  p.logits = static_cast<const bf16*>(logits); p.ld = ld;
  p.token = reinterpret_cast<int64_t*>(token); p.out = reinterpret_cast<int64_t*>(out); p.out_ld = out_ld; p.columns = columns;
  p.cursor = reinterpret_cast<int64_t*>(cursor); p.pos = reinterpret_cast<int64_t*>(pos);
  p.positions = reinterpret_cast<int64_t*>(positions);
  for (int i = 0; i < rings; ++i) {
    if (caps[i] < 1) return TTCD_ERR_ARG;
    p.slot[i] = reinterpret_cast<int64_t*>(slots[i]); p.kv_len[i] = kv_lens[i]; p.cap[i] = caps[i];
  }
  p.best = static_cast<unsigned long long*>(best); p.turns = turns;
  p.B = B; p.V = V; p.rings = rings;
  return launch_dependent(decode_pick_kernel, dim3(PICK_SPLIT, B), dim3(PICK_THREADS), 0, static_cast<cudaStream_t>(stream_ptr), p);
}

// layers (up to 32): k, v [B, rows, heads x dim] with batch and row strides in elements -> rings [B, capacity, heads x dim] (batch
// stride ring_b, rows contiguous); rows <= capacity, start >= rows.  All addresses 16-byte aligned, all strides and the row
// length (elements) multiples of 8.  record: per layer k, v, rk, rv, sk_b, sk_r, sv_b, sv_r, ring_b, rows, capacity as int64.
TTCD_EXPORT int ttcd_ring_load(const long long* record, int layers, int B, int row_elems, long long start, void* stream_ptr) {
  using namespace ttcd;
  if (layers < 1 || layers > RING_LAYERS || B < 1 || B > 65535 || row_elems < 8 || row_elems % 8 != 0) return TTCD_ERR_ARG;
  RingParams p;
  p.start = start;
  p.vecs = row_elems / 8;
  int64_t most = 0;
  for (int i = 0; i < layers; ++i) {
    const long long* r = record + 11 * i;
    for (int j = 0; j < 4; ++j) if (r[j] == 0 || r[j] % 16 != 0) return TTCD_ERR_ARG;
    for (int j = 4; j < 9; ++j) if (r[j] < 0 || r[j] % 8 != 0) return TTCD_ERR_ARG;
    if (r[9] < 0 || r[10] < 1 || r[9] > r[10] || r[10] > 0x3fffffff || start < r[9]) return TTCD_ERR_ARG;
    RingLayer& L = p.layer[i];
    L.k = reinterpret_cast<const bf16*>(r[0]); L.v = reinterpret_cast<const bf16*>(r[1]);
    L.rk = reinterpret_cast<bf16*>(r[2]); L.rv = reinterpret_cast<bf16*>(r[3]);
    L.sk_b = r[4]; L.sk_r = r[5]; L.sv_b = r[6]; L.sv_r = r[7]; L.ring_b = r[8];
    L.rows = static_cast<int>(r[9]); L.cap = static_cast<int>(r[10]);
    most = most > r[9] ? most : r[9];
  }
  if (most == 0) return TTCD_OK;
  if (most * p.vecs > 0x40000000) return TTCD_ERR_SIZE;
  const int64_t blocks = (most * p.vecs + RING_THREADS * RING_VECS - 1) / (RING_THREADS * RING_VECS);
  const dim3 grid(static_cast<unsigned>(blocks < 4096 ? blocks : 4096), 2 * layers, B);
  ring_load_kernel<<<grid, RING_THREADS, 0, static_cast<cudaStream_t>(stream_ptr)>>>(p);
  return static_cast<int>(cudaGetLastError());
}
