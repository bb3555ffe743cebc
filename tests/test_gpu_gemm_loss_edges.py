"""fp32 outputs of the GEMM (stored and added in place) at tile edges, the chunking of the linear cross-entropy, and the
cross-entropy's gradient next to untouched logits."""
import pytest
import torch

from ttcd_b200.ops import cuda

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,batch", [(128, 128, 64, 1), (129, 132, 72, 1), (300, 260, 136, 3), (1000, 516, 640, 1), (128, 1028, 64, 2)])
@pytest.mark.parametrize("a_t,b_t", [(False, True), (True, False)])
def test_fp32_output_and_accumulation(M, N, K, batch, a_t, b_t):
    torch.manual_seed(M + N)
    pad = lambda n: -(-n // 8) * 8                                                     # noqa: E731  (operand rows: 16 bytes)
    a = torch.randn(batch, K, pad(M), device=DEV).bfloat16()[..., :M].transpose(-1, -2) if a_t else torch.randn(batch, M, pad(K), device=DEV).bfloat16()[..., :K]
    b = torch.randn(batch, N, pad(K), device=DEV).bfloat16()[..., :K].transpose(-1, -2) if b_t else torch.randn(batch, K, pad(N), device=DEV).bfloat16()[..., :N]
    want = a.double() @ b.double()
    guard = torch.full((batch + 1, M, N), 7.0, device=DEV)                             # what lies behind the output stays
    out = guard[:batch]
    cuda.gemm(a, b, out_dtype=torch.float32, out=out)
    bound = 2.0 ** -20 * K                                                             # K products of size ~1 summed in fp32
    assert (out.double() - want).abs().max() <= bound
    cuda.gemm(a, b, out_dtype=torch.float32, out=out, beta=1.0, c_in=out, alpha=0.5)
    assert (out.double() - 1.5 * want).abs().max() <= 2 * bound
    other = torch.randn_like(out)
    sep = torch.empty_like(out)
    cuda.gemm(a, b, out_dtype=torch.float32, out=sep, beta=2.0, c_in=other)            # another addend: the reading epilogue
    assert (sep.double() - (want + 2 * other.double())).abs().max() <= 2 * bound
    assert (guard[batch] == 7.0).all()


@pytest.mark.parametrize("n,hidden,chunks", [(128, 64, 8), (600, 1024, 8), (5003, 2048, 8), (65536, 1024, 8), (65536, 960, 32), (2560, 2048, 1),
                                             (24000, 4096, 8), (1, 1024, 8)])
def test_lm_head_chunks_cover_the_rows_and_stay_bounded(n, hidden, chunks):
    rows = cuda._lce_chunk_rows(n, hidden, chunks)
    assert rows % 128 == 0 and rows > 0
    assert rows <= max(-(-n // 128) * 128 if chunks == 1 else 0, 2560 if chunks <= 8 else 0, int(1.25 * n / chunks) + 128)


@pytest.mark.parametrize("n,hidden", [(5003, 2048), (8192, 2048), (16384, 2048), (40000, 1024), (65536, 960)])
def test_more_chunks_than_the_default_take_less_memory(n, hidden):
    rows = [cuda._lce_chunk_rows(n, hidden, chunks) for chunks in (9, 16, 32, 64)]
    assert all(r <= 1.25 * n / c + 128 for r, c in zip(rows, (9, 16, 32, 64)))
    assert rows == sorted(rows, reverse=True) and rows[-1] < cuda._lce_chunk_rows(n, hidden, 8)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,vocab,offset", [(3, 1000, 0), (130, 128, 0), (7, 4096, 8), (5, 1000, 4)])
@pytest.mark.parametrize("smoothing,z", [(0.0, 0.0), (0.1, 1e-3)])
def test_cross_entropy_gradient_beside_the_logits(rows, vocab, offset, smoothing, z):
    torch.manual_seed(rows)
    store = (3 * torch.randn(rows * vocab + offset, device=DEV)).bfloat16()
    leaf = store.requires_grad_()
    logits = leaf[offset:].view(rows, vocab)                # offset 4: 8-byte aligned only
    labels = torch.randint(0, vocab, (rows,), device=DEV)
    labels[0] = -100
    kept = logits.detach().clone()
    loss = cuda.cross_entropy(logits, labels, label_smoothing=smoothing, z_loss=z)
    grads = [torch.autograd.grad(loss * s, leaf, retain_graph=True)[0][offset:].view(rows, vocab).double() for s in (1.0, 3.0, 1.0)]
    assert torch.equal(logits, kept) and torch.equal(grads[0], grads[2])
    x = kept.double().requires_grad_()
    lse = torch.logsumexp(x, -1)
    valid = labels != -100
    per = lse - (1 - smoothing) * x.gather(1, labels.clamp_min(0)[:, None])[:, 0] - smoothing * x.mean(-1) + z * lse ** 2
    want_loss = (per * valid).sum() / valid.sum()
    (want,) = torch.autograd.grad(want_loss, x)
    assert abs(float(loss) - float(want_loss)) < 1e-4 * abs(float(want_loss))
    # one rounding to bf16 of values whose exponentials carry a few fp32 roundings; scaled by 3: one more
    assert ((grads[0] - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()
    assert ((grads[1] - 3 * want).abs() <= 2.0 ** -7 * 3 * want.abs() + 1e-6).all()


@pytest.mark.gpu
@pytest.mark.parametrize("linear", [False, True])
def test_loss_gradient_is_linear_in_what_arrives(linear):
    """A learned weight of the loss (``create_graph``) and several weights at once (``is_grads_batched``)."""
    torch.manual_seed(1)
    x = torch.randn(128, 128 if linear else 512, device=DEV).bfloat16().requires_grad_()
    w = torch.randn(512, 128, device=DEV).bfloat16()
    labels = torch.randint(0, 512, (128,), device=DEV)
    loss = lambda: cuda.linear_cross_entropy(x, labels, w) if linear else cuda.cross_entropy(x, labels)     # noqa: E731
    (one,) = torch.autograd.grad(loss(), x)
    weight = torch.tensor(2.0, device=DEV, requires_grad=True)
    (twice,) = torch.autograd.grad(loss() * weight, x, create_graph=True)
    assert torch.equal(twice, 2 * one)                       # doubling rounds nothing
    (by_weight,) = torch.autograd.grad(twice.float().sum(), weight)
    want = one.double().sum()
    # d(sum of the gradient) / d weight = the sum, of bf16 values that the library adds in fp32 and rounds to bf16
    assert abs(float(by_weight.double() - want)) <= 2.0 ** -8 * float(want.abs()) + 2.0 ** -20 * float(one.double().abs().sum())
    (several,) = torch.autograd.grad(loss(), x, torch.tensor([1.0, 4.0], device=DEV), is_grads_batched=True)
    assert torch.equal(several[0], one) and torch.equal(several[1], 4 * one)


@pytest.mark.gpu
@pytest.mark.parametrize("batch,M,N,K", [
    (1, 128, 128, 64), (1, 300, 1024, 3072), (1, 448, 2056, 520), (1, 1024, 1032, 2328), (1, 130, 19000, 72),          # 64 or 128 wide
    (1, 2048, 1024, 200), (1, 6002, 1024, 136), (3, 1030, 1160, 264), (1, 129, 136, 1000),                             # 128 wide
    (1, 3832, 1024, 200), (2, 1100, 2050 // 8 * 8, 128)])                                                              # 256 wide
@pytest.mark.parametrize("a_t,b_t,out", [(False, True, "bf16"), (False, False, "bf16"), (True, False, "fp32"), (True, True, "bf16+c")])
def test_gemm_of_every_tile_width_against_float64(batch, M, N, K, a_t, b_t, out):
    """Shapes on both sides of the rule for the tile's width, with remainders of rows, columns and K, every operand order."""
    torch.manual_seed(M + N)
    M, N = M // 8 * 8 if a_t else M, N // 8 * 8
    mk = lambda r, c, t: (torch.randn(batch, c, r, device=DEV).bfloat16().transpose(1, 2) if t                         # noqa: E731
                          else torch.randn(batch, r, c, device=DEV).bfloat16())
    a, b = mk(M, K, a_t), mk(K, N, b_t)
    c = torch.randn(batch, M, N, device=DEV).bfloat16() if out == "bf16+c" else None
    got = cuda.gemm(a, b, out_dtype=torch.float32 if out == "fp32" else torch.bfloat16, c_in=c, beta=0.0 if c is None else 1.0).double()
    want = a.double() @ b.double() + (0.0 if c is None else c.double())
    # K / 16 accumulation steps, each cut within an ulp or two (2^-23, 2^-22) of a partial sum of up to 4 sqrt(K); then one rounding to bf16
    bound = max(K, 16) / 16 * 2.0 ** -22 * 4 * K ** 0.5 + (0.0 if out == "fp32" else want.abs() * 2.0 ** -8)
    assert got.shape == want.shape and ((got - want).abs() <= bound).all(), float(((got - want).abs() - bound).max())


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(12000, 192, 64), (12000, 192, 2048), (9600, 136, 72), (20000, 1088, 64), (20000, 1088, 520), (16500, 320, 64),
                                   (20000, 168, 136), (20000, 1056, 64)])
@pytest.mark.parametrize("out", ["bf16", "fp32", "bf16+c"])
def test_gemm_with_several_tiles_per_cta_and_an_odd_number_of_stores_in_one(M, N, K, out):
    """A tile of one store (64 columns wide, or cut there by the edge) is followed by another tile of the same CTA, whose first store
    must not go through the staging buffer that the former one is read from.  Short products, so that the stores follow one another."""
    torch.manual_seed(M + N + K)
    a, b = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    c = torch.randn(1, M, N, device=DEV).bfloat16() if out == "bf16+c" else None
    want = a.double() @ b.double().T + (0.0 if c is None else c[0].double())
    # K / 16 accumulation steps, each cut within an ulp or two (2^-23, 2^-22) of a partial sum of up to 4 sqrt(K); then one rounding to bf16
    bound = max(K, 16) / 16 * 2.0 ** -22 * 4 * K ** 0.5 + (0.0 if out == "fp32" else want.abs() * 2.0 ** -8)
    for _ in range(5):
        got = cuda.gemm(a, b.T, out_dtype=torch.float32 if out == "fp32" else torch.bfloat16, c_in=c, beta=0.0 if c is None else 1.0)
        err = (got.view(M, N).double() - want).abs() - bound
        assert (err <= 0).all(), float(err.max())
