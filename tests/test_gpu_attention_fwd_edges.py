"""Attention forward against float64 where its schedule changes: one or two query tiles per CTA, lengths around multiples of
the 128-row tile and 128-key block, windows shorter than a block and across several, keys ahead of the queries, packed
sequences whose tiles see different ranges, a running maximum that keeps growing, a negative scale."""
import pytest
import torch

from ttcd_b200.ops import cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _reference(q, k, v, windows, scale, starts=None):
    B, Tq, H, D = q.shape
    Tk, G = k.shape[1], H // k.shape[2]
    kf, vf = (t.double().repeat_interleave(G, dim=2) for t in (k, v))
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), kf) * scale
    qpos = torch.arange(Tk - Tq, Tk, device=DEV)[:, None]
    key = torch.arange(Tk, device=DEV)[None, :]
    out = []
    for w in windows:
        vis = (key <= qpos) if w is None else (key <= qpos) & (key > qpos - w)
        if starts is not None:
            vis = vis & (key >= starts[:, None])
        x = s.masked_fill(~vis, float("-inf"))
        out.append((torch.einsum("bhqk,bkhd->bqhd", torch.softmax(x, -1), vf), torch.logsumexp(x, -1)))
    return out


def _check(got, want, lse, want_lse, mass=None):
    # P is rounded to bf16 before P V (relative 2^-9 per term, averaging out over the keys), the output once more.  With `mass`
    # (P |V|): every term's rounding at its largest (2^-8) and of one sign, which a few dominant keys come near
    err = (got.double() - want).abs()
    slack = 2.0 ** -7 * want.abs() + 2.0 ** -7 * want.square().mean().sqrt() if mass is None else 2.0 ** -8 * (want.abs() + mass)
    assert (err <= slack + 1e-3).all(), float(err.max())
    assert (got.double() - want).norm() <= 4e-3 * want.norm() + 1e-6
    assert (lse.double() - want_lse).abs().max() <= 1e-4


@pytest.mark.parametrize("D,H,HK", [(128, 2, 1), (64, 3, 3)])
@pytest.mark.parametrize("Tq,ahead", [(128, 0), (129, 0), (255, 0), (256, 0), (257, 0), (384, 0), (641, 0), (130, 100), (300, 1), (256, 515)])
@pytest.mark.parametrize("w_t,w_s", [(None, None), (1, 1), (64, 63), (128, 1), (129, 128), (400, 131), (10000, 256), (512, 512)])
def test_forward_schedule_edges(D, H, HK, Tq, ahead, w_t, w_s):
    torch.manual_seed(Tq + ahead)
    q = 2 * torch.randn(2, Tq, H, D, device=DEV)
    q = (q * torch.linspace(0.5, 3, Tq, device=DEV)[None, :, None, None]).bfloat16()     # later rows: sharper, more rescaling
    k = (torch.randn(2, Tq + ahead, HK, D, device=DEV)).bfloat16()
    v = torch.randn(2, Tq + ahead, HK, D, device=DEV).bfloat16()
    scale = D ** -0.5
    dual = w_s is not None
    _, o_t, o_s, lse_t, lse_s = cuda.attn_forward(q, k, v, w_t, w_s if dual else w_t, scale, dual)
    want = _reference(q, k, v, [w_t, w_s] if dual else [w_t], scale)
    _check(o_t, want[0][0], lse_t, want[0][1])
    if dual:
        _check(o_s, want[1][0], lse_s, want[1][1])


@pytest.mark.parametrize("form", [1, 2])                     # long, short: wherever the rule would send the call
@pytest.mark.parametrize("D,H,HK", [(128, 2, 1), (64, 3, 3)])
@pytest.mark.parametrize("Tq,ahead", [(128, 0), (129, 0), (257, 0), (384, 0), (641, 0), (300, 1), (256, 515), (1027, 0)])
@pytest.mark.parametrize("w_t,w_s", [(None, None), (None, 200), (1, 1), (64, 63), (128, 1), (129, 128), (400, 131), (10000, 256)])
def test_both_forms_at_the_edges(D, H, HK, Tq, ahead, w_t, w_s, form):
    torch.manual_seed(Tq + ahead)
    q = 2 * torch.randn(2, Tq, H, D, device=DEV)
    q = (q * torch.linspace(0.5, 3, Tq, device=DEV)[None, :, None, None]).bfloat16()
    k, v = (torch.randn(2, Tq + ahead, HK, D, device=DEV).bfloat16() for _ in range(2))
    dual = w_s is not None
    _, o_t, o_s, lse_t, lse_s = cuda.attn_forward(q, k, v, w_t, w_s if dual else w_t, D ** -0.5, dual, form=form)
    windows = [w_t, w_s] if dual else [w_t]
    want, mass = _reference(q, k, v, windows, D ** -0.5), _reference(q, k, v.abs(), windows, D ** -0.5)
    _check(o_t, want[0][0], lse_t, want[0][1], mass[0][0])
    if dual:
        _check(o_s, want[1][0], lse_s, want[1][1], mass[1][0])


@pytest.mark.parametrize("form", [1, 2])
@pytest.mark.parametrize("D", [64, 128])
def test_both_forms_packed_negative_scale_and_not_a_number(D, form):
    torch.manual_seed(D)
    bounds, T = (0, 1, 2, 130, 383, 384, 900), 900
    q, k, v = (torch.randn(1, T, h, D, device=DEV).bfloat16() for h in (2, 2, 2))
    seg = cuda.segment_bounds(torch.tensor(bounds, device=DEV), T)
    _, o_t, o_s, lse_t, lse_s = cuda.attn_forward(q, k, v, 300, 140, -0.3, True, seg, form=form)
    want = _reference(q, k, v, [300, 140], -0.3, seg[0].long())
    _check(o_t, want[0][0], lse_t, want[0][1])
    _check(o_s, want[1][0], lse_s, want[1][1])
    k[0, 17, 0] = float("nan")
    _, o, _, _, _ = cuda.attn_forward(q, k, v, None, None, D ** -0.5, False, form=form)
    assert o[0, 17:, 0].isnan().any(-1).all() and not o[:, :17].isnan().any() and not o[:, :, 1].isnan().any()


@pytest.mark.parametrize("B,T,H,D,w", [(160, 128, 1, 128, None), (40, 300, 16, 64, None), (4, 384, 16, 128, None), (1, 20000, 1, 64, 64),
                                       (1, 512, 16, 128, None), (1, 513, 16, 128, None), (1, 300, 4, 64, None)])
def test_forms_agree_on_both_sides_of_the_rule(B, T, H, D, w):
    torch.manual_seed(T)
    q, k, v = (torch.randn(B, T, H, D, device=DEV).bfloat16() for _ in range(3))
    run = lambda form: cuda.attn_forward(q, k, v, w, None if w is None else w // 2, D ** -0.5, w is not None, form=form)      # noqa: E731
    rule, long, short = run(0), run(1), run(2)
    assert any(torch.equal(rule[1], f[1]) for f in (long, short))
    for a, b in zip(long[1:], short[1:]):
        if a is not None:            # each within its bound of the exact values (see above)
            assert (a.float() - b.float()).norm() <= 8e-3 * b.float().norm()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bounds", [(0, 128, 640), (0, 500, 513, 641), (0, 1, 2, 130, 400), (0, 255, 256, 900)])
def test_forward_packed_sequences(D, bounds):
    torch.manual_seed(bounds[-1])
    T = bounds[-1]
    q, k, v = (torch.randn(1, T, h, D, device=DEV).bfloat16() for h in (2, 1, 1))
    seg = cuda.segment_bounds(torch.tensor(bounds, device=DEV), T)
    _, o_t, o_s, lse_t, lse_s = cuda.attn_forward(q, k, v, 300, 140, D ** -0.5, True, seg)
    want = _reference(q, k, v, [300, 140], D ** -0.5, seg[0].long())
    _check(o_t, want[0][0], lse_t, want[0][1])
    _check(o_s, want[1][0], lse_s, want[1][1])


@pytest.mark.parametrize("D", [64, 128])
def test_forward_negative_scale_and_not_a_number(D):
    torch.manual_seed(D)
    q, k, v = (torch.randn(1, 300, 2, D, device=DEV).bfloat16() for _ in range(3))
    _, o, _, lse, _ = cuda.attn_forward(q, k, v, None, None, -0.3, False)
    want = _reference(q, k, v, [None], -0.3)
    _check(o, want[0][0], lse, want[0][1])
    k[0, 17, 0] = float("nan")                               # one key of one head: every row that sees it is lost, none before
    _, o, _, _, _ = cuda.attn_forward(q, k, v, None, None, D ** -0.5, False)
    assert o[0, 17:, 0].isnan().any(-1).all() and not o[:, :, 1].isnan().any()
