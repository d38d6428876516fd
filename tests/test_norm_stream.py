"""The residual sum + RMS norm of many rows (the streaming form) against float64 and against the form of a block a row; the
experts' combine with the same inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows,hidden", [(250001, 4), (30000, 36), (1300, 1024), (513, 2052), (2048, 5120), (1025, 8192)])
@pytest.mark.parametrize("top_k,weighted", [(0, False), (1, False), (2, True), (8, True)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_norm_and_combine(rows, hidden, top_k, weighted, dtype):
    from hi_b200.kernels import ops

    g = torch.Generator(device=DEV).manual_seed(rows + hidden + top_k)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x0, delta, w = rnd(rows, hidden), rnd(rows, hidden).to(dtype), (1 + 0.1 * rnd(hidden)).to(dtype)
    delta2 = rnd(rows, hidden).to(torch.bfloat16) if top_k == 0 else None
    kw = {"delta2": delta2, "x_scale": 0.5 if top_k == 2 else 1.0}
    total = x0.double() * kw["x_scale"] + delta.double() + (delta2.double() if delta2 is not None else 0.0)
    if top_k:
        routed, slot = rnd(rows * top_k, hidden), torch.randperm(rows * top_k, device=DEV, generator=g).to(torch.int32)
        rw = torch.rand(rows * top_k, device=DEV, generator=g) if weighted else None
        kw.update(routed=routed, slot_of_entry=slot, top_k=top_k, routed_weight=rw)
        parts = routed.double()[slot.long()].view(rows, top_k, hidden)
        if weighted:
            parts = parts * rw.double().view(rows, top_k, 1)
        total = total + parts.sum(1)
        combined = ops.moe_combine(routed, slot, delta, rows, top_k, rw)
        assert float((combined.double() - parts.sum(1) - delta.double()).abs().max()) <= 8 * 2.0 ** -24 * float(total.abs().max() + 8)
    want = total / torch.sqrt((total * total).mean(1, keepdim=True) + 1e-5) * w.double()
    for post in (False, True):
        x = x0.clone()
        y, y32 = ops.add_rmsnorm(x, delta, w, 1e-5, torch.bfloat16, also_f32=True, post=post, **kw)
        # sums of up to eleven terms and of the row's squares, each within a few 2^-24
        assert float((y32.double() - want).abs().max()) <= 2e-6 * float(want.abs().max())
        assert torch.equal(y, y32.to(torch.bfloat16))
        assert torch.equal(x, y32) if post else float((x.double() - total).abs().max()) <= 1e-6 * float(total.abs().max())
    one = torch.cat([ops.add_rmsnorm(x0[i: i + 500].clone(), delta[i: i + 500].contiguous(), w, 1e-5, torch.float32, x_scale=kw["x_scale"],
                                     delta2=None if delta2 is None else delta2[i: i + 500].contiguous()) for i in range(0, min(rows, 5000), 500)])
    many = ops.add_rmsnorm(x0.clone(), delta, w, 1e-5, torch.float32, x_scale=kw["x_scale"], delta2=delta2)
    many = many[: len(one)]
    assert float((one - many).abs().max()) <= 2e-6 * float(one.abs().max())      # the order of a row's squares differs


@pytest.mark.parametrize("rows,hidden", [(2048, 2048), (1905, 2048), (513, 8188), (2050, 5120)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_norm_alone(rows, hidden, out_dtype):
    """Nothing to add: from 3.9 million numbers on the streaming form, which leaves the stream as it is, to the bit."""
    from hi_b200.kernels import ops

    g = torch.Generator(device=DEV).manual_seed(rows)
    x0, w = torch.randn(rows, hidden, device=DEV, generator=g), 1 + 0.1 * torch.randn(hidden, device=DEV, generator=g)
    x0[7, 5], x0[9] = float("inf"), float("nan")               # each stays in its row
    fine = torch.ones(rows, dtype=torch.bool, device=DEV)
    fine[7] = fine[9] = False
    want = x0.double() / torch.sqrt((x0.double() ** 2).mean(1, keepdim=True) + 1e-5) * w.double()
    x = x0.clone()
    y, y32 = ops.add_rmsnorm(x, None, w, 1e-5, out_dtype, also_f32=True)
    assert torch.equal(x.view(torch.int32), x0.view(torch.int32))
    assert float((y32 - want)[fine].abs().max()) <= 2e-6 * float(want[fine].abs().max())
    assert torch.equal(y[fine], y32[fine].to(out_dtype)) and bool(torch.isnan(y[9]).all()) and bool(torch.isnan(y[7, 5]))
