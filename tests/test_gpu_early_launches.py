"""Launches that may start before the kernel in front of them has ended: the same bits on both sides of the rule, and after everything
that may stand in front of one on its stream."""
import pytest
import torch

from ttcd_b200.ops import cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SMS = 148


def _norm(x, w):
    return cuda.rmsnorm(x, w, 1e-6)


@pytest.mark.parametrize("rows", [8 * 2 * SMS - 1, 8 * 2 * SMS, 8 * 2 * SMS + 1])            # eight rows per CTA, two CTAs per SM
def test_a_row_has_the_same_bits_on_both_sides_of_the_rule(rows):
    torch.manual_seed(rows)
    x, w = torch.randn(rows, 512, device=DEV).bfloat16(), torch.randn(512, device=DEV).bfloat16()
    parts = torch.cat([_norm(x[i:i + 500], w) for i in range(0, rows, 500)])
    assert torch.equal(_norm(x, w), parts)
    a, b = x, torch.randn(1024, 512, device=DEV).bfloat16()
    pieces = torch.cat([cuda.gemm(a[i:i + 128 * 4], b.T).view(-1, 1024) for i in range(0, rows - rows % 512, 512)])
    assert torch.equal(cuda.gemm(a, b.T).view(-1, 1024)[:pieces.shape[0]], pieces)


@pytest.mark.parametrize("seq,heads,dim", [(128, 2 * SMS, 64), (129, 2 * SMS, 64), (300, 8, 128), (300, 296, 128)])
def test_attention_on_both_sides_of_the_rule(seq, heads, dim):
    """Heads in one call and one by one: the last CTAs of a large call and the first ones of a small call do the same work."""
    torch.manual_seed(seq + heads)
    q, k, v = (torch.randn(1, seq, heads, dim, device=DEV).bfloat16() for _ in range(3))
    for form in (1, 2):
        whole = cuda.attn_forward(q, k, v, 100, None, dim ** -0.5, False, form=form)[1]
        for h in (0, heads - 1):
            one = cuda.attn_forward(*(t[:, :, h:h + 1].contiguous() for t in (q, k, v)), 100, None, dim ** -0.5, False, form=form)[1]
            assert torch.equal(whole[:, :, h:h + 1], one)


def _chain(x, w, buf):
    """Copies, memsets and small launches one after the other; each reads what the one before it wrote."""
    buf.zero_()
    buf.copy_(x)                                                     # a copy in front of a small launch
    y = _norm(buf, w)
    buf.copy_(y)
    y = cuda.gemm(buf, torch.eye(buf.shape[1], device=DEV, dtype=torch.bfloat16)).view_as(buf)
    buf.zero_()                                                      # y was read from it by a launch that may still run
    return _norm(y, w)


def test_small_launches_after_copies_and_memsets_and_under_capture():
    torch.manual_seed(0)
    x, w = torch.randn(300, 1024, device=DEV).bfloat16(), torch.randn(1024, device=DEV).bfloat16()
    want = _norm(_norm(x.clone(), w).clone(), w)
    buf = torch.empty_like(x)
    for _ in range(20):
        assert torch.equal(_chain(x, w, buf), want)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        first = _norm(x, w)                                          # the first node
        here = torch.cuda.current_stream()
        side.wait_stream(here)
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000)
            second = _norm(first, w)
        third = _chain(x, w, buf)
        here.wait_stream(side)
        joined = cuda.rmsnorm(second, w, 1e-6, residual=third)       # after a join of two streams
    for _ in range(5):
        for t in (first, second, third, joined):
            t.fill_(7.0)
        graph.replay()
        assert torch.equal(third, want) and torch.equal(second, want) and torch.equal(joined, cuda.rmsnorm(want, w, 1e-6, residual=want))


def test_a_small_launch_waits_for_an_event_of_another_stream():
    torch.manual_seed(1)
    x, w = torch.randn(300, 1024, device=DEV).bfloat16(), torch.randn(1024, device=DEV).bfloat16()
    want = _norm(x.clone(), w)
    side = torch.cuda.Stream()
    late = torch.zeros_like(x)
    for _ in range(10):
        late.zero_()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.cuda._sleep(500_000)
            late.copy_(x)
        before = _norm(x, w)                                         # the kernel in front, on this stream
        torch.cuda.current_stream().wait_stream(side)
        assert torch.equal(_norm(late, w), want) and torch.equal(before, want)
        late.record_stream(side)
