"""Products with several weights side by side, a residual or SwiGLU against the separate ops: the same bits."""
import pytest
import torch

from ttcd_b200 import _native as nv
from ttcd_b200.ops import cuda

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("M,K,sizes", [(128, 64, (64, 64, 64)), (300, 136, (192, 64, 64)), (1000, 1024, (512, 256, 256)), (2000, 72, (2048, 128, 136)),
                                       (700, 520, (256, 320))])
def test_weights_in_pieces_make_the_same_product(M, K, sizes):
    torch.manual_seed(M)
    x = torch.randn(M, K, device=DEV).bfloat16()
    ws = [torch.randn(n, K, device=DEV).bfloat16() for n in sizes]
    w = torch.cat(ws)
    res = torch.randn(M, w.shape[0], device=DEV).bfloat16()
    guard = torch.full((M + 1, w.shape[0]), 7.0, device=DEV).bfloat16()          # what lies behind the output stays
    for r in (None, res):
        out = guard[:M]
        nv.call("ttcd_gemm_pieces", nv.ptr(x), nv.ptr(ws[0]), nv.ptr(ws[1]), nv.ptr(ws[2] if len(ws) > 2 else None), nv.ptr(out), nv.ptr(r),
                nv.i64(M), nv.i64(w.shape[0]), nv.i64(K), nv.i64(K), nv.i64(K), nv.i64(w.shape[0]), nv.i64(sizes[0]), nv.i64(sizes[1]),
                nv.i32(0), nv.stream_ptr())
        want = cuda.gemm(x, w.transpose(0, 1)).view(M, -1)
        assert torch.equal(out, want if r is None else want + r)
        assert (guard[M] == 7).all()


@pytest.mark.parametrize("M,K,N", [(128, 64, 128), (300, 1024, 3072), (1000, 264, 136), (3000, 128, 2056), (129, 72, 1000)])
def test_swiglu_on_the_product(M, K, N):
    torch.manual_seed(N)
    x = torch.randn(M, K, device=DEV).bfloat16()
    g, u = (torch.randn(N, K, device=DEV).bfloat16() for _ in range(2))
    g *= 100 * K ** -0.5                                                        # saturated gates among them
    out = torch.empty(M, N, device=DEV).bfloat16()
    nv.call("ttcd_gemm_pieces", nv.ptr(x), nv.ptr(g), nv.ptr(u), nv.ptr(None), nv.ptr(out), nv.ptr(None), nv.i64(M), nv.i64(N), nv.i64(K),
            nv.i64(K), nv.i64(K), nv.i64(N), nv.i64(0), nv.i64(0), nv.i32(1), nv.stream_ptr())
    want = cuda.swiglu(cuda.gemm(x, g.transpose(0, 1)).view(M, N), cuda.gemm(x, u.transpose(0, 1)).view(M, N))
    assert torch.equal(out, want)


@pytest.mark.parametrize("M,K", [(300, 960), (700, 960), (3000, 64), (9001, 960)])
def test_weights_in_pieces_that_leave_no_wide_tile(M, K):
    """960 + 320 + 320 columns: tiles are 64 wide, and from 6 rows of tiles on a CTA has more than one of them."""
    torch.manual_seed(M)
    sizes = (960, 320, 320)
    x = torch.randn(M, K, device=DEV).bfloat16()
    ws = [torch.randn(n, K, device=DEV).bfloat16() for n in sizes]
    res = torch.randn(M, 1600, device=DEV).bfloat16()
    want = cuda.gemm(x, torch.cat(ws).transpose(0, 1)).view(M, -1)
    for r in (None, res) * 3:
        out = torch.empty(M, 1600, device=DEV).bfloat16()
        nv.call("ttcd_gemm_pieces", nv.ptr(x), nv.ptr(ws[0]), nv.ptr(ws[1]), nv.ptr(ws[2]), nv.ptr(out), nv.ptr(r), nv.i64(M), nv.i64(1600),
                nv.i64(K), nv.i64(K), nv.i64(K), nv.i64(1600), nv.i64(960), nv.i64(320), nv.i32(0), nv.stream_ptr())
        assert torch.equal(out, want if r is None else want + r)
