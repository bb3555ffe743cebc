"""Where no gradient is recorded an op may run its forward without the autograd machinery around it (``cuda._apply``).  A
program must not see the difference: a tracer records the op, not the memory it happened to write, and what comes back is
what ``Function.apply`` returns.  ``_Twice`` does its work behind the tracer's back, as a kernel launch does."""
import pytest
import torch

from ttcd_b200.ops import cuda


class _Twice(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        y = torch.empty_like(x)
        y.numpy()[...] = x.detach().numpy() * 2
        return y

    @staticmethod
    def backward(ctx, g):
        return 2 * g


@pytest.mark.filterwarnings("ignore")          # (the tracer says that it cannot follow numpy)
def test_a_tracer_records_the_op():
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: cuda._apply(_Twice, x) + 0, (torch.ones(3),), check_trace=False)
        assert any(n.kind() == "prim::PythonOp" for n in traced.graph.nodes())
        assert torch.equal(traced(torch.full((3,), 5.0)), torch.full((3,), 10.0))


def test_gradients_are_recorded_where_they_are_on():
    x = torch.ones(3, requires_grad=True)
    with torch.no_grad():
        assert not cuda._apply(_Twice, x).requires_grad
    assert torch.equal(torch.autograd.grad(cuda._apply(_Twice, x).sum(), x)[0], torch.full((3,), 2.0))


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
def test_rmsnorm_hands_its_input_through_as_a_tensor_of_its_own(mode):
    x = torch.randn(5, 256, device="cuda:0").bfloat16().requires_grad_()
    w = torch.ones(256, device="cuda:0", dtype=torch.bfloat16)
    with mode():
        _, through = cuda.rmsnorm(x, w, 1e-6, prenorm=True)
    assert through is not x and not through.requires_grad and through.data_ptr() == x.data_ptr()
    y, through = cuda.rmsnorm(x, w, 1e-6, prenorm=True)
    (g,) = torch.autograd.grad((y.float().sum() + 2 * through.float().sum()), x)
    assert g.shape == x.shape and bool(g.isfinite().all())
