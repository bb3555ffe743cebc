"""Ops that split their work in one way for large calls and in another for small ones: the two give the same values, bit by
bit, so a large call is compared with the same rows in small calls (weight gradients, which sum over the rows, with float64).
Sizes lie on both sides of each rule; the small route itself is compared with the oracle in the ops' own tests."""
import pytest
import torch

from ttcd_b200 import ops
from ttcd_b200.ops import cuda

DEV, BF = "cuda:0", torch.bfloat16


@pytest.mark.gpu
@pytest.mark.parametrize("D,H,HK", [(128, 4, 2), (128, 8, 4), (128, 7, 4), (128, 16, 16), (128, 3, 0), (64, 15, 5), (64, 16, 17)])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("rows", [1600, 8200, 32771])
def test_head_norm_and_rotary(D, H, HK, norm, rows):
    torch.manual_seed(rows)
    q, k = torch.randn(1, rows, H, D, device=DEV).to(BF), torch.randn(1, rows, HK, D, device=DEV).to(BF)
    w = [(1 + 0.2 * torch.randn(D, device=DEV)).to(BF) if norm else None for _ in range(2)]
    cos, sin = (torch.randn(rows, D // 2, device=DEV).to(BF) for _ in range(2))
    dq, dk = torch.randn_like(q), torch.randn_like(k)

    def run(a, b):
        qs, ks = (t[:, a:b].contiguous().requires_grad_() for t in (q, k))
        ws = [None if t is None else t.clone().requires_grad_() for t in w]
        out = cuda.qk_norm_rope(qs, ks, *ws, 1e-6, cos, sin, a)
        leaves = [qs] + ([ks] if HK else []) + [t for t in ws if t is not None]
        grads = torch.autograd.grad(out if HK else out[:1], leaves, (dq[:, a:b], dk[:, a:b])[:2 if HK else 1])
        return out, grads

    out, grads = run(0, rows)
    parts = [run(a, min(a + 1000, rows)) for a in range(0, rows, 1000)]
    for i in range(2):
        assert torch.equal(out[i], torch.cat([p[0][i] for p in parts], 1))
    for i in range(2 if HK else 1):
        assert torch.equal(grads[i], torch.cat([p[1][i] for p in parts], 1))
    if norm:
        n = 2 if HK else 1
        for x, dy, g in zip((q, k)[:n], (dq, dk)[:n], grads[n:]):
            xd, d = x[0].double(), dy[0].double()
            lo, hi, c, s = d[..., :D // 2], d[..., D // 2:], cos.double()[:, None], sin.double()[:, None]
            d = torch.cat([lo * c + hi * s, hi * c - lo * s], -1)
            want = (d * xd * (xd.square().mean(-1, keepdim=True) + 1e-6).rsqrt()).sum((0, 1))
            # fp32 sums of rows * heads terms of size ~1.5 in blocks (random signs), one rounding to bf16
            assert ((g.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * (rows * x.shape[2]) ** 0.5).all()


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 520, 1024, 1032, 3072])
@pytest.mark.parametrize("total", [8 << 20, 40 << 20])
def test_swiglu(d, total):
    rows = total // d + 3
    torch.manual_seed(d)
    gate_up = (2 * torch.randn(rows, 2 * d, device=DEV)).to(BF)
    whole = cuda.swiglu_packed(gate_up)
    assert torch.equal(whole, torch.cat([cuda.swiglu_packed(gate_up[a:a + 500]) for a in range(0, rows, 500)]))
    g, u = gate_up[-700:, :d].double(), gate_up[-700:, d:].double()
    want = torch.nn.functional.silu(g) * u
    # one rounding to bf16; the fp32 exponential's error is far below it
    assert ((whole[-700:].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-30).all()


@pytest.mark.gpu
@pytest.mark.parametrize("V,rows", [(8192, 149), (8200, 149), (32000, 160), (32003, 160), (70000, 460)])
@pytest.mark.parametrize("smoothing,z,l2", [(0.0, 0.0, 0.0), (0.1, 1e-3, 0.0), (0.0, 0.0, 1e-3)])
def test_cross_entropy_rows(V, rows, smoothing, z, l2):
    torch.manual_seed(V)
    ld = -(-V // 8) * 8
    logits = (3 * torch.randn(rows, ld, device=DEV)).to(BF)[:, :V]
    labels = torch.randint(0, V, (rows,), device=DEV)
    labels[1] = -100
    scale = torch.full((1,), 0.25, device=DEV)

    def run(a, b):
        grad = torch.zeros(b - a, ld, dtype=BF, device=DEV)[:, :V]
        return cuda._ce_rows(logits[a:b], labels[a:b], scale, -100, True, smoothing, z, l2, grad=grad), grad

    loss, grad = run(0, rows)
    parts = [run(a, min(a + 40, rows)) for a in range(0, rows, 40)]
    assert torch.equal(loss, torch.cat([p[0] for p in parts])) and torch.equal(grad, torch.cat([p[1] for p in parts]))


@pytest.mark.gpu
@pytest.mark.parametrize("N,K", [(3071, 1024), (3072, 1024), (3072, 1032), (4097, 2048), (9000, 256), (5000, 4096)])
def test_one_row_times_weight(N, K):
    torch.manual_seed(N)
    x, w = torch.randn(1, K, device=DEV).to(BF), (torch.randn(N, K, device=DEV) * K ** -0.5).to(BF)
    got, want = cuda.gemm(x, w.t(), alpha=0.5).double(), 0.5 * x.double() @ w.double().t()
    # fp32 accumulation (K terms of size ~K^-1/2) and one rounding to bf16
    assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -22 * K ** 0.5).all()


@pytest.mark.parametrize("D,pairs", [(64, 1), (64, 2), (64, 3), (64, 4), (64, 8), (128, 1), (128, 2), (128, 4), (128, 7)])
@pytest.mark.parametrize("heads", [1, 5, 8, 64, 400])
@pytest.mark.parametrize("Tk", [1, 127, 300, 2345, 70001])
def test_key_ranges_of_a_decode_step(D, pairs, heads, Tk):
    splits = cuda._decode_splits(heads, pairs, Tk, D)
    turn = 8 * (32 // (D // 8)) * (8 if pairs <= 4 else 4)                  # warps x keys per load x loads
    assert 1 <= splits <= -(-Tk // turn) and (splits == 1 or splits * heads <= 148 * (2 if pairs <= 2 else 1))
