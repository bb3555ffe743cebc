"""AdamW against float64 where its accesses change: both gradient types, arrays that are not aligned for four elements at a
time, lengths with a remainder, skipped steps, without the bf16 copy."""
import pytest
import torch

from ttcd_b200.ops import cuda

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 4, 1027, 300002])
@pytest.mark.parametrize("grad_dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("off", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 0, 2)])           # of p, m, v; grad; bf16 copy
@pytest.mark.parametrize("skip,copy", [(None, True), (0, True), (1, True), (0, False)])
def test_adamw_step(n, grad_dtype, off, skip, copy):
    torch.manual_seed(n)
    lr, b1, b2, eps, wd, clip = torch.tensor([1e-2, 0.9, 0.95, 1e-8, 0.1, 0.5]).tolist()      # as the kernel gets them: fp32 values
    step = 3
    store = lambda o, dtype: torch.rand(n + o + 4, device=DEV).to(dtype)                 # noqa: E731  (four more: what lies behind)
    bufs = [store(off[0], torch.float32), store(off[0], torch.float32), store(off[0], torch.float32), store(off[1], grad_dtype),
            store(off[2], torch.bfloat16)]
    bufs[3].sub_(0.5)
    kept = [b.clone() for b in bufs]
    offs = (off[0], off[0], off[0], off[1], off[2])
    p, m, v, g, pb = (b[o:o + n] for b, o in zip(bufs, offs))
    pd, md, vd, gd = (t.double() for t in (p, m, v, g))
    cuda.adamw_step(p, g, m, v, pb if copy else None, lr=lr, beta1=b1, beta2=b2, eps=eps, weight_decay=wd, step=step,
                    coef=torch.tensor([clip], device=DEV), skip=None if skip is None else torch.tensor([skip], dtype=torch.int32, device=DEV))
    for b, k, o in zip(bufs, kept, offs):                                                # neighbours stay
        assert torch.equal(b[:o], k[:o]) and torch.equal(b[o + n:], k[o + n:])
    assert torch.equal(bufs[3], kept[3])
    if skip:
        assert all(torch.equal(b, k) for b, k in zip(bufs, kept))
        return
    gd = gd * clip
    mw, vw = b1 * md + (1 - b1) * gd, b2 * vd + (1 - b2) * gd * gd
    update = lr / (1 - b1 ** step) * mw / (vw.sqrt() / (1 - b2 ** step) ** 0.5 + eps)
    want = pd * (1 - lr * wd) - update
    # values of size ~1 through at most a dozen fp32 roundings; the moving averages' terms may cancel, their errors do not
    scale = lr / (1 - b1 ** step) * (md + gd.abs()) / (vw.sqrt() / (1 - b2 ** step) ** 0.5 + eps)
    assert ((m.double() - mw).abs() <= 2.0 ** -22 * (md + gd.abs())).all() and ((v.double() - vw).abs() <= 2.0 ** -21 * vw).all()
    assert ((p.double() - want).abs() <= 2.0 ** -22 * pd.abs() + 2.0 ** -20 * scale).all()
    assert torch.equal(pb, p.bfloat16()) if copy else torch.equal(bufs[4], kept[4])
