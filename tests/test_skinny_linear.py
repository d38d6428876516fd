"""Products of a few bfloat16 rows against the same in float64: edges of the kernel's tiles (16 rows of the weight, 8 tokens,
32 of K), each of its forms, rows that are a slice of a wider matrix, and what is left to the library."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n_out,k", [(1, 8), (15, 40), (17, 2048), (2368, 64), (2369, 328), (4737, 264), (6657, 128), (48, 4104)])
@pytest.mark.parametrize("tokens", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_against_float64(n_out, k, tokens, out_dtype):
    from hi_b200.kernels import ops
    from hi_b200.parts.linear import linear

    g = torch.Generator(device=DEV).manual_seed(n_out + k)
    wide = torch.randn(tokens, k + 24, device=DEV, generator=g).to(torch.bfloat16)
    x, w = wide[:, 8: 8 + k], (torch.randn(n_out, k, device=DEV, generator=g) * k ** -0.5).to(torch.bfloat16)
    bias = torch.randn(n_out, device=DEV, generator=g).to(torch.bfloat16)
    want = x.double() @ w.double().t()
    got = ops.skinny_linear(x, w, out_dtype)
    if tokens > 8 and n_out > 2368:
        assert got is None
        return
    # float32 sums of k exact products of size one in all: a few 2^-24; bfloat16 results: 2^-9 of the value
    tol = 2e-6 if out_dtype == torch.float32 else 2.0 ** -8
    assert float((got.double() - want).abs().max()) <= tol * float(want.abs().max())
    got = linear(x, w, out_dtype=out_dtype, bias=bias)
    want = want + bias.double()
    assert got.dtype == out_dtype and float((got.double() - want).abs().max()) <= tol * float(want.abs().max())


def test_what_is_left_to_the_library():
    from hi_b200.kernels import ops
    from hi_b200.parts.linear import linear

    x, w = torch.randn(4, 72, device=DEV).to(torch.bfloat16), torch.randn(33, 72, device=DEV).to(torch.bfloat16)
    flat = torch.randn(4 * 72 + 1, device=DEV).to(torch.bfloat16)
    for a, b in ((x[:, :68], w[:, :68].contiguous()), (x[:, 4:68], w[:, :64].contiguous()), (x, w.t().contiguous().t()),
                 (torch.randn(17, 72, device=DEV).to(torch.bfloat16), w), (flat[1:].view(4, 72), w), (x[:0], w),
                 (x.t().contiguous().t(), w)):
        assert ops.skinny_linear(a, b, torch.bfloat16) is None
        got, want = linear(a, b), a.double() @ b.double().t()
        assert got.shape == want.shape and (not got.numel() or float((got.double() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max()))
    with pytest.raises(Exception):
        linear(x, w[:, :64].contiguous())


@pytest.mark.parametrize("n_out,k,tokens,taken", [
    (4736, 8192, 8, True), (4736, 8200, 2, False), (4737, 4088, 1, True), (4737, 4096, 1, False), (4737, 4104, 2, True),
    (4737, 2056, 8, True), (6657, 2048, 8, True), (6657, 2056, 5, False), (6657, 8192, 4, True),
    (6657, 8200, 2, False), (8193, 1024, 2, False), (8193, 1032, 8, True),
    (16383, 5128, 8, False), (16384, 1016, 3, False), (16384, 5128, 8, True), (16400, 8200, 2, False), (65544, 2048, 1, True),
    (65544, 2056, 2, False), (2368, 8200, 16, True)])
def test_where_the_kernel_is_the_faster_one(n_out, k, tokens, taken):
    """The ends of the ranges that the kernel takes; rows long enough that its ring of loads goes round."""
    from hi_b200.kernels import ops

    g = torch.Generator(device=DEV).manual_seed(n_out + k)
    x = torch.randn(tokens, k, device=DEV, generator=g).to(torch.bfloat16)
    w = (torch.randn(n_out, k, device=DEV, generator=g) * k ** -0.5).to(torch.bfloat16)
    got = ops.skinny_linear(x, w, torch.float32)
    assert (got is not None) == taken
    if taken:
        want = x.double() @ w.double().t()
        assert float((got.double() - want).abs().max()) <= 2e-6 * float(want.abs().max())


def test_operands_on_the_host_are_refused_and_gradients_kept():
    from hi_b200.parts.linear import linear

    x, w = torch.randn(4, 72, device=DEV).to(torch.bfloat16), torch.randn(33, 72, device=DEV).to(torch.bfloat16)
    for weight, bias in ((w.cpu(), None), (w, torch.zeros(33, dtype=torch.bfloat16))):
        with pytest.raises(RuntimeError):
            linear(x, weight, bias=bias)
    w.requires_grad_()
    linear(x, w).float().sum().backward()
    want = x.double().sum(0).expand_as(w)                # four terms in float32, rounded to bfloat16: 2^-9 of the value
    assert float((w.grad.double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())


def test_tangents_and_transforms_go_through_the_library():
    from hi_b200.parts.linear import linear

    x, dx = (torch.randn(3, 4, 72, device=DEV).to(torch.bfloat16) for _ in range(2))
    w = torch.randn(33, 72, device=DEV).to(torch.bfloat16)
    close = lambda got, want: float((got.double() - want).abs().max()) <= 2.0 ** -8 * float(want.abs().max())
    assert close(torch.func.vmap(lambda row: linear(row, w))(x), x.double() @ w.double().t())
    y, dy = torch.func.jvp(lambda t: linear(t, w), (x[0],), (dx[0],))
    assert close(y, x[0].double() @ w.double().t()) and close(dy, dx[0].double() @ w.double().t())
    with torch.autograd.forward_ad.dual_level():
        out = linear(torch.autograd.forward_ad.make_dual(x[1], dx[1]), w)
        assert close(torch.autograd.forward_ad.unpack_dual(out).tangent, dx[1].double() @ w.double().t())
