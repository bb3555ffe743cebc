"""The decode step's kernels against float64: attention of a few (query row, head) pairs over a key/value cache (its pair
counts, partly filled rings, windows, key counts around the sizes of a turn and of a split) and the products of up to 16 rows
with a weight (row, column and K remainders)."""
import pytest
import torch

from ttcd_b200 import _native
from ttcd_b200.models import IPTTCDv9Config, IPTTCDv9ForCausalLM
from ttcd_b200.models.decoding import GraphDecoder
from ttcd_b200.models.layers import WindowKVCache
from ttcd_b200.ops import cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _attention64(q, k, v, window, n):
    """q [B,Tq,H,D] at the end of the first n keys, bottom-right causal."""
    B, Tq, H, D = q.shape
    G = H // k.shape[2]
    kf, vf = (t[:, :n].double().repeat_interleave(G, dim=2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), kf) * D ** -0.5
    qpos = torch.arange(n - Tq, n, device=q.device)[:, None]
    key = torch.arange(n, device=q.device)[None, :]
    vis = (key <= qpos) if window is None else (key <= qpos) & (key > qpos - window)
    return torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s.masked_fill(~vis, float("-inf")), -1), vf)


@pytest.mark.parametrize("B,Tq,Tk,H,HK,D,W,filled", [
    (1, 1, 1, 1, 1, 128, None, None), (2, 1, 127, 4, 4, 64, None, None), (1, 1, 128, 4, 2, 128, None, None),
    (3, 1, 129, 6, 2, 64, 100, None), (1, 2, 2049, 8, 2, 128, 500, None), (1, 1, 8192, 16, 8, 128, None, 1501),
    (5, 1, 640, 15, 5, 64, None, 1), (2, 8, 999, 2, 2, 128, 64, None), (1, 1, 70001, 2, 1, 64, None, None),
    (2, 1, 300, 14, 2, 128, None, 299), (1, 2, 1000, 4, 1, 64, None, 257)])
def test_decode_attention_against_float64(B, Tq, Tk, H, HK, D, W, filled):
    assert Tq * (H // HK) <= 8
    torch.manual_seed(Tk)
    q, k, v = (torch.randn(B, t, h, D, device=DEV).bfloat16() for t, h in ((Tq, H), (Tk, HK), (Tk, HK)))
    q = q * 2                                                # a sharper softmax: the running max moves
    n = Tk if filled is None else filled
    if filled is not None:                                   # rows past the fill count must not be read
        k[:, n:], v[:, n:] = float("nan"), float("nan")
    kv_len = None if filled is None else torch.tensor([n], dtype=torch.int32, device=DEV)
    got = cuda.attn_small_q(q, k, v, W, None, kv_len).double()
    turns = torch.zeros(B * HK, dtype=torch.int32, device=DEV)          # the splits merged in the same launch, twice
    for _ in range(2):
        one = cuda.attn_small_q(q, k, v, W, None, kv_len, turns).double()
        assert (turns == 0).all() and (one - got).abs().max() <= 2.0 ** -8 * got.abs().max()
    want = _attention64(q, k, v, W, n)
    # fp32 sums (scores up to ~40: absolute error below 1e-5, so is the probabilities' relative one) and one rounding to bf16
    bound = want.abs() * 2.0 ** -8 + 1e-4
    assert ((got - want).abs() <= bound).all(), float(((got - want).abs() - bound).max())


@pytest.mark.parametrize("Tq,H,HK,D", [(1, 4, 2, 128), (3, 2, 1, 64)])
def test_decode_attention_takes_a_query_at_any_address(Tq, H, HK, D):
    torch.manual_seed(Tq)
    k, v = (torch.randn(1, 300, HK, D, device=DEV).bfloat16() for _ in range(2))
    q = torch.randn(Tq * H * D + 1, device=DEV).bfloat16()[1:].view(1, Tq, H, D)           # contiguous, 2-byte aligned
    got, want = cuda.attn_small_q(q, k, v).double(), _attention64(q, k, v, None, 300)
    assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 1e-4).all()


def test_decode_attention_counts_its_launches():
    q, k = torch.randn(1, 1, 4, 64, device=DEV).bfloat16(), torch.randn(1, 300, 2, 64, device=DEV).bfloat16()
    before = _native.launch_count
    cuda.attn_small_q(q, k, k)
    apart = _native.launch_count
    cuda.attn_small_q(q, k, k, turns=torch.zeros(2, dtype=torch.int32, device=DEV))
    assert (apart - before, _native.launch_count - apart) == (2, 1)          # with and without a merge of its own


@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (1, 1024, 2048), (3, 129, 72), (8, 6144, 1024), (8, 1001, 3072), (9, 130, 264),
                                   (16, 4096, 1024), (16, 20000, 520), (5, 151936, 1024)])
def test_few_rows_times_weight_against_float64(M, N, K):
    torch.manual_seed(N + K)
    x = torch.randn(M, K, device=DEV).bfloat16()
    w = (torch.randn(N, K, device=DEV) * K ** -0.5).bfloat16()
    got = cuda.gemm(x, w.transpose(0, 1), alpha=0.5).double()
    want = 0.5 * x.double() @ w.double().t()
    # fp32 accumulation (K terms of size ~K^-1/2) and one rounding to bf16
    bound = want.abs() * 2.0 ** -8 + 2.0 ** -22 * K ** 0.5
    assert got.shape == (M, N) and ((got - want).abs() <= bound).all(), float(((got - want).abs() - bound).max())


@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (3, 130, 264), (8, 1001, 1024), (9, 256, 2048), (16, 3072, 1032)])
@pytest.mark.parametrize("norm,swiglu,residual", [(True, False, False), (True, True, False), (False, False, True), (False, True, True)])
def test_few_rows_with_norm_swiglu_residual(M, N, K, norm, swiglu, residual):
    """What rides along with the product rounds where the separate ops round."""
    torch.manual_seed(N + K)
    x = torch.randn(M, K, device=DEV).bfloat16()
    nw = (1 + 0.1 * torch.randn(K, device=DEV)).bfloat16()
    w = (torch.randn(2 * N if swiglu else N, K, device=DEV) * K ** -0.5).bfloat16()
    res = torch.randn(M, N, device=DEV).bfloat16() if residual else None
    got = cuda.gemv(x, w, norm=(nw, 1e-6) if norm else None, swiglu=swiglu, residual=res).double()
    xd = x.double()
    if norm:
        xd = (xd * (xd.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * nw.double()).bfloat16().double()
    y = (xd @ w.double().t()).bfloat16().double()
    if swiglu:
        y = (torch.nn.functional.silu(y[:, :N]) * y[:, N:]).bfloat16().double()
    want = y if res is None else (y + res.double())
    # up to four roundings to bf16 (each may fall to the neighbour) on values and summands of size ~1
    bound = 2.0 ** -7 * (want.abs() + y.abs()) + 2.0 ** -7
    assert ((got - want).abs() <= bound).all(), float(((got - want).abs() - bound).max())
    assert (got - want).abs().mean() < 2.0 ** -9


@pytest.mark.parametrize("batch,heads,kv_heads,dim,prompt,window", [(1, 4, 2, 128, 240, 256), (3, 5, 5, 64, 40, 64), (16, 8, 2, 64, 130, None)])
def test_fused_decode_step_matches_module_by_module(batch, heads, kv_heads, dim, prompt, window):
    """The captured step of a model (fused projections, ring writes, wrapped rings) against the same step run through the
    modules: same roundings, sums in another order."""
    torch.manual_seed(3)
    cfg = IPTTCDv9Config(hidden_size=256, num_hidden_layers=2, num_heads=heads, num_kv_heads=kv_heads, head_dim=dim,
                         intermediate_size=520, vocab_size=1000, window_size=window, max_position_embeddings=512, ttt_mode=False,
                         ttt_layers=[], qk_norm=True, tie_word_embeddings=False)
    model = IPTTCDv9ForCausalLM(cfg).to(DEV, torch.bfloat16).eval()
    ids = torch.randint(0, 1000, (batch, prompt), device=DEV)
    cache = WindowKVCache()
    with torch.no_grad():
        model(input_ids=ids, past_key_values=cache, use_cache=True, logits_to_keep=1)
    dec = GraphDecoder(model, cache, 40)
    assert dec.fused is not None
    first, steps = ids[:, -1:], 40
    assert window is None or prompt + steps > window         # the rings wrap and are full
    dec.token.copy_(first)
    got = []
    for _ in range(steps):
        dec.graph.replay()
        got.append(dec.last_logits.clone())
    tokens, rings = dec.out[:, :steps].clone(), [(k.clone(), v.clone()) for k, v in dec.cache.layers.values()]
    dec.fused = None                                         # module by module, fed the same tokens
    dec.load(cache)
    feed = torch.cat([first, tokens], dim=1)
    with torch.no_grad():
        for i in range(steps):
            dec.token.copy_(feed[:, i:i + 1])
            want = dec._logits().float()
            dec.cache.advance()
            err = (got[i].float() - want).norm() / want.norm()
            assert err < 0.02, (i, float(err))
    for (k, v), (rk, rv) in zip(rings, dec.cache.layers.values()):
        for a, b in ((k, rk), (v, rv)):
            assert (a.float() - b.float()).norm() / b.float().norm() < 0.02


@pytest.mark.parametrize("B,V", [(1, 1), (2, 7), (3, 4099), (16, 32000), (1, 151936)])
def test_next_token_and_the_move_of_the_rings(B, V):
    """Against torch.argmax (ties to the first, a NaN above all) and the arithmetic of the cache's own advance."""
    torch.manual_seed(V)
    logits = torch.randn(B, V, device=DEV).bfloat16()
    logits[0, V // 2:] = logits[0].max()                      # ties
    logits[0, V - 1] = -0.0
    if B > 1:
        logits[1, V // 3] = float("nan")
    if B > 2:
        logits[2] = float("-inf")
    i64 = lambda *v: torch.tensor(v, dtype=torch.int64, device=DEV)          # noqa: E731
    token, out, cursor, pos = i64(*[-1] * B).view(B, 1), torch.full((B, 3), -1, dtype=torch.int64, device=DEV), i64(1), i64(511)
    positions, scratch = i64(*[511] * B).view(B, 1), torch.zeros(8 * B + 1, dtype=torch.int64, device=DEV)
    rings = [(c, i64(0), torch.zeros(1, dtype=torch.int32, device=DEV)) for c in (512, 1000, 7)]
    want = logits.float().argmax(-1)
    for step in range(3):                                    # the last one finds its column past the end
        cuda.decode_pick(logits, token, out, cursor, pos, positions, rings, scratch)
        at = 512 + step
        assert (token.view(-1) == want).all() and int(cursor) == 2 + step and int(pos) == at and (positions == at).all()
        for c, slot, kv_len in rings:
            assert int(slot) == at % c and int(kv_len) == min(at + 1, c)
    assert (out[:, 0] == -1).all() and (out[:, 1] == want).all() and (out[:, 2] == want).all() and int(scratch[0]) == 0


@pytest.mark.parametrize("B,HK,D,cap,n,start", [(1, 8, 128, 64, 64, 64), (2, 5, 64, 100, 37, 250), (3, 1, 64, 9, 9, 13), (1, 2, 128, 4096, 1, 1)])
def test_ring_load_against_indexed_copies(B, HK, D, cap, n, start):
    torch.manual_seed(n)
    wide = torch.randn(B, n, 3 * HK * D, device=DEV).bfloat16()               # k and v as columns of one projection, and on their own
    pairs = [(wide[..., :HK * D].view(B, n, HK, D), wide[..., HK * D:2 * HK * D].view(B, n, HK, D)),
             tuple(torch.randn(B, n, HK, D, device=DEV).bfloat16() for _ in range(2)),
             tuple(torch.randn(B * n * HK * D + 1, device=DEV).bfloat16()[1:].view(B, n, HK, D) for _ in range(2))]       # misaligned
    rings = [tuple(torch.full((B, cap, HK, D), 7.0, device=DEV).bfloat16() for _ in range(2)) for _ in pairs]
    assert cuda.ring_load([(*p, *r) for p, r in zip(pairs, rings)], start) == [2]
    rows = torch.arange(start - n, start, device=DEV) % cap
    for src, ring in zip(pairs[:2], rings):
        for s, r in zip(src, ring):
            want = torch.full_like(r, 7.0)
            want.index_copy_(1, rows, s)
            assert torch.equal(r, want)
    assert (rings[2][0] == 7).all()
