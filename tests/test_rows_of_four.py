"""Kernels that take four or eight neighbouring channels a thread where the rows allow it: against float64 at the edges of what
they take, and where the general kernels stay (odd sizes, columns that start off their bytes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kvh,dim,vdim,taps,shift", [(4, 2, 128, 128, 4, 0), (2, 2, 4, 8, 4, 4), (3, 1, 132, 64, 4, 0), (2, 1, 256, 200, 4, 8),
                                                           (2, 2, 64, 128, 3, 0), (2, 1, 30, 64, 4, 0), (2, 2, 64, 64, 4, 1), (1, 1, 260, 64, 4, 0)])
@pytest.mark.parametrize("head_decay", [False, True])
@pytest.mark.parametrize("lens", [[1, 7, 2], [3, 250, 13, 1]])
def test_delta_prep(heads, kvh, dim, vdim, taps, shift, head_decay, dt, lens):
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(dim + vdim + taps)
    slots = ([2, 0, 3, 1] if len(lens) <= 4 else list(range(len(lens)))[::-1])[: len(lens)]
    n, c = sum(lens), 2 * kvh * dim + heads * vdim
    rnd = lambda *s: torch.randn(*s, generator=g)
    off = taps + (4 if taps == 4 else 1)                             # where the convolution's rows start in the state
    proj = rnd(n, shift + c + heads + (-(shift + c + heads)) % 4).to(dt)
    w, state, per = rnd(c, taps), rnd(max(4, len(lens)), off + (taps - 1) * c + (-(off + (taps - 1) * c)) % 4), heads if head_decay else heads * dim
    pre, bias, a_log = rnd(n, per).to(dt), rnd(per), 0.3 * rnd(heads)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    seq = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(torch.int32)
    d = lambda t: t.to(DEV)
    got = ops.delta_prep(d(proj), shift, shift + c, d(w), d(state), off, d(pre), d(bias), d(a_log), d(cu), d(seq),
                         d(torch.tensor(slots, dtype=torch.int32)), heads, kvh, dim, vdim, head_decay=head_decay)
    P, y = proj.double(), []
    for s, slot in enumerate(slots):
        rows = torch.cat([state[slot, off: off + (taps - 1) * c].double().view(taps - 1, c), P[int(cu[s]): int(cu[s + 1]), shift: shift + c]])
        conv = sum(w[:, j].double() * rows[j: j + lens[s]] for j in range(taps))
        y.append(conv * torch.sigmoid(conv))
    y = torch.cat(y)
    unit = lambda t: t / (t.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
    q, k, v = y[:, : kvh * dim].view(n, kvh, dim), y[:, kvh * dim: 2 * kvh * dim].view(n, kvh, dim), y[:, 2 * kvh * dim:]
    rate, x = torch.exp(a_log.double()).view(1, heads, 1), pre.double() + bias.double()
    x = (x.view(n, heads, 1).expand(n, heads, dim) if head_decay else x.view(n, heads, dim))
    want = (unit(q).reshape(n, -1) * dim ** -0.5, unit(k).reshape(n, -1), v, torch.sigmoid(P[:, shift + c: shift + c + heads]),
            torch.exp(-rate * torch.nn.functional.softplus(x)).reshape(n, -1))
    for a, b, name in zip(got, want, ("q", "k", "v", "beta", "decay")):
        # a few float32 roundings of 6e-8 in sums of four products, and of the length's sum over at most 260 squares
        assert float((a.cpu().double() - b).abs().max() / b.abs().max()) < 2e-6, name


# two tokens a warp (rows of up to 128 and of more, borders of requests inside a warp's), eight, and one where the step is of single tokens
@pytest.mark.parametrize("heads,kvh,dim,vdim,lens", [(16, 16, 128, 128, [3, 250, 13, 1]), (8, 8, 132, 40, [1, 700, 3]), (16, 4, 40, 36, [300, 215]),
                                                     (16, 16, 64, 96, [5, 2000, 703]), (32, 16, 128, 100, [2001]), (16, 16, 128, 128, [1] * 260)])
def test_delta_prep_of_many_tokens(heads, kvh, dim, vdim, lens):
    test_delta_prep(heads, kvh, dim, vdim, 4, 0, False, torch.bfloat16, lens)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("n,heads,vdim,shift,pad", [(5, 4, 128, 0, 0), (3, 2, 36, 4, 4), (2, 3, 200, 0, 8), (2, 1, 256, 8, 0), (3, 2, 132, 4, 0), (9, 3, 64, 0, 4),
                                                    # the general kernel: an odd stride, rows not of whole fours, off their bytes, too long, many short ones
                                                    (5, 4, 128, 0, 3), (3, 2, 130, 0, 0), (2, 2, 64, 1, 3), (1, 2, 260, 0, 0), (2501, 4, 32, 0, 0),
                                                    (3, 2, 4, 4, 0), (3, 5, 32, 0, 0)])
def test_delta_out_norm(n, heads, vdim, shift, pad, silu, dt):
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(vdim + n)
    rnd = lambda *s: torch.randn(*s, generator=g)
    o, wide, w = rnd(n, heads * vdim), rnd(n, shift + heads * vdim + pad).to(dt), rnd(vdim).to(dt)
    gate = wide[:, shift: shift + heads * vdim]
    got = ops.delta_out_norm(o.to(DEV), wide.to(DEV)[:, shift: shift + heads * vdim], w.to(DEV), 1e-5, vdim, dt, gate_silu=silu)
    x, z = o.double().view(n, heads, vdim), gate.double().reshape(n, heads, vdim)
    want = x / (x.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() * (z * torch.sigmoid(z) if silu else torch.sigmoid(z))
    err = float((got.cpu().double().view_as(want) - want).abs().max() / want.abs().max())
    assert err < (2 ** -8 if dt == torch.bfloat16 else 2e-6), err       # one rounding of the result; a few of float32


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,heads,dim", [(5, 16, 128), (1, 1, 8), (37, 3, 24), (4, 5, 12), (300, 2, 1)])
def test_head_gate(n, heads, dim, dt):
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(n + dim)
    x, wide = torch.randn(n, heads, dim, generator=g).to(dt), 3.0 * torch.randn(n, heads + 5, generator=g).to(dt)
    got = ops.head_gate(x.to(DEV), wide.to(DEV)[:, 2: 2 + heads])
    want = x.double() * torch.sigmoid(wide[:, 2: 2 + heads].double()).unsqueeze(2)
    err = float((got.cpu().double() - want).abs().max() / want.abs().max())
    assert err < (2 ** -8 if dt == torch.bfloat16 else 1e-6), err
