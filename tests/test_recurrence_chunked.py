"""The recurrences sixteen tokens at a time (portions of prompts), against the same recurrences token after token in
float64: partial chunks, one-token requests beside portions, sizes around the kernels' tiles of 16 rows and columns."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# outputs and states, largest error over largest value: sums of at most 128 float32 products (sqrt(128) 2^-24 = 7e-7 of their
# length) whose factors carry a few roundings of 6e-8 each, over memories of some dozens of tokens: 3e-6 with room
TOL = 3e-6
LENS = [1, 16, 130, 17, 15, 2]


def close(got, want, what):
    err = float((got.double().cpu() - want.double().cpu()).abs().max() / want.abs().max().clamp_min(1e-30))
    assert err <= TOL, (what, err)


def tables(lens):
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32)
    slots = torch.randperm(len(lens) + 2, generator=torch.Generator().manual_seed(1))[: len(lens)].to(torch.int32)
    return cu, slots


@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("heads,kvh,dim,vdim", [(4, 2, 128, 128), (2, 2, 1, 1), (3, 3, 16, 16), (2, 1, 17, 33), (4, 4, 64, 15),
                                                (2, 1, 65, 17), (6, 3, 96, 40), (1, 1, 112, 130), (9, 9, 127, 129)])
def test_delta_rule_and_plain(heads, kvh, dim, vdim, plain):
    from hi_b200.kernels import ops

    assert ops._chunked_recurrence(sum(LENS), len(LENS), dim)
    g = torch.Generator().manual_seed(dim)
    n = sum(LENS)
    rnd = lambda *s: torch.randn(*s, generator=g)
    q = (F.normalize(rnd(n, kvh, dim), dim=-1) * dim ** -0.5).reshape(n, -1)
    k = F.normalize(rnd(n, kvh, dim), dim=-1).reshape(n, -1)
    v, beta = rnd(n, heads * vdim), torch.rand(n, heads, generator=g)
    decay = torch.exp(-torch.exp(2.0 * rnd(n, heads * dim) - 2.0))       # from almost one to far underflow in a chunk
    decay[5, :3] = 0.0
    cu, slots = tables(LENS)
    state = rnd(len(LENS) + 2, heads * dim * vdim + 3)
    dev = state.to(DEV)
    o = ops.delta_recurrence(q.to(DEV), k.to(DEV), v.to(DEV), None if plain else beta.to(DEV), decay.to(DEV), dev, cu.to(DEV),
                             slots.to(DEV), heads, kvh, dim, vdim, plain=plain)
    wide = lambda t: t.double().view(n, kvh, dim).repeat_interleave(heads // kvh, dim=1)
    qd, kd, vd, gd = wide(q), wide(k), v.double().view(n, heads, vdim), decay.double().view(n, heads, dim)
    for s, slot in enumerate(slots.tolist()):
        S = state[slot, : heads * dim * vdim].double().view(heads, dim, vdim)
        want = []
        for t in range(int(cu[s]), int(cu[s + 1])):
            S = S * gd[t][:, :, None]
            u = vd[t] if plain else beta[t].double()[:, None] * (vd[t] - torch.einsum("hdv,hd->hv", S, kd[t]))
            S = S + kd[t][:, :, None] * u[:, None, :]
            want.append(torch.einsum("hdv,hd->hv", S, qd[t]).reshape(-1))
        close(o[int(cu[s]): int(cu[s + 1])], torch.stack(want), f"request {s}")
        close(dev[slot, : heads * dim * vdim], S.reshape(-1), f"state {s}")
        assert torch.equal(dev[slot, heads * dim * vdim:].cpu(), state[slot, heads * dim * vdim:])
    for slot in set(range(len(LENS) + 2)) - set(slots.tolist()):
        assert torch.equal(dev[slot].cpu(), state[slot])


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,dim,vdim", [(4, 128, 128), (3, 16, 15), (2, 33, 16), (1, 1, 1), (2, 96, 47), (10, 64, 129)])
def test_mlstm(heads, dim, vdim, dt):
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(dim)
    n, off = sum(LENS), 3
    proj = (0.5 * torch.randn(n, off + heads * (2 * dim + vdim) + 1, generator=g)).to(dt)
    keep, take = torch.rand(n, heads, generator=g), torch.rand(n, heads, generator=g)
    cu, slots = tables(LENS)
    floats = ops.mlstm_state_floats(heads, dim, vdim)
    state = 0.3 * torch.randn(len(LENS) + 2, floats, generator=g)
    dev = state.to(DEV)
    o, nq = ops.mlstm_recurrence(proj.to(DEV), off, off + heads * dim, off + 2 * heads * dim, dim ** -0.5, keep.to(DEV),
                                 take.to(DEV), dev, cu.to(DEV), slots.to(DEV), heads, dim, vdim)
    p = proj.double()
    q, k = (p[:, off + i * heads * dim: off + (i + 1) * heads * dim].view(n, heads, dim) for i in (0, 1))
    v = torch.cat([p[:, off + 2 * heads * dim: -1].view(n, heads, vdim), torch.ones(n, heads, 1, dtype=torch.float64)], dim=2)
    for s, slot in enumerate(slots.tolist()):
        S = state[slot, : heads * (vdim + 1) * dim].double().view(heads, vdim + 1, dim)
        want = []
        for t in range(int(cu[s]), int(cu[s + 1])):
            S = keep[t].double().view(-1, 1, 1) * S + (take[t].double()[:, None] * v[t])[:, :, None] * k[t][:, None, :]
            want.append(torch.einsum("hvd,hd->hv", S, q[t]) * dim ** -0.5)
        want, rows = torch.stack(want), slice(int(cu[s]), int(cu[s + 1]))
        close(o[rows], want[:, :, :vdim], f"request {s}")
        close(nq[rows], want[:, :, vdim], f"n.q of request {s}")
        close(dev[slot, : heads * (vdim + 1) * dim], S.reshape(-1), f"state {s}")
        assert torch.equal(dev[slot, heads * (vdim + 1) * dim:].cpu(), state[slot, heads * (vdim + 1) * dim:])


def test_what_is_not_finite_stays_with_later_tokens_and_its_column():
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(0)
    n, heads, dim, vdim = 200, 2, 64, 48
    q, k = (F.normalize(torch.randn(n, heads, dim, generator=g), dim=-1).reshape(n, -1).to(DEV) for _ in range(2))
    v, beta = torch.randn(n, heads * vdim, generator=g).to(DEV), torch.rand(n, heads, generator=g).to(DEV)
    decay = (0.5 + 0.5 * torch.rand(n, heads * dim, generator=g)).to(DEV)
    cu, slots = torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    call = lambda: ops.delta_recurrence(q, k, v, beta, decay, torch.zeros(1, heads * dim * vdim, device=DEV), cu, slots, heads,
                                        heads, dim, vdim)
    clean = call()
    v[70, 5] = float("nan")
    got = call()
    assert bool(torch.isnan(got[70:, 5]).all())
    other = torch.ones_like(got, dtype=torch.bool)
    other[70:, 5] = False
    assert torch.equal(got[other], clean[other])


@pytest.mark.parametrize("plain", [False, True])
def test_the_end_of_the_range(plain):
    """Finite values and states above bfloat16's largest number (3.39e38): their own columns as in float64, the others as
    without them. Keys of half a unit and decays below a half keep the float32 sums themselves in range."""
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(7)
    n, heads, dim, vdim, top = 200, 2, 64, 48, 3.4e38
    q, k = (0.5 * F.normalize(torch.randn(n, heads, dim, generator=g), dim=-1).reshape(n, -1) for _ in range(2))
    v, beta = torch.randn(n, heads * vdim, generator=g), torch.rand(n, heads, generator=g)
    decay = 0.1 + 0.3 * torch.rand(n, heads * dim, generator=g)
    cu, slots = torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    state = torch.zeros(1, heads * dim * vdim)

    def call():
        s = state.to(DEV)
        o = ops.delta_recurrence(q.to(DEV), k.to(DEV), v.to(DEV), None if plain else beta.to(DEV), decay.to(DEV), s, cu, slots, heads,
                                 heads, dim, vdim, plain=plain)
        return o.cpu(), s.cpu()

    clean, clean_state = call()
    v[70, 5], v[71, vdim + 3] = top, -top                 # head 0 column 5, head 1 column 3
    state.view(heads, dim, vdim)[1, 2, 9] = top
    got, got_state = call()
    S, want = state.double().view(heads, dim, vdim).clone(), []
    for t in range(n):
        kt, qt, vt = (x[t].double().view(heads, -1) for x in (k, q, v))
        S = S * decay[t].double().view(heads, dim, 1)
        u = vt if plain else beta[t].double()[:, None] * (vt - torch.einsum("hdv,hd->hv", S, kt))
        S = S + kt[:, :, None] * u[:, None, :]
        want.append(torch.einsum("hdv,hd->hv", S, qt).reshape(-1))
    want, touched = torch.stack(want), torch.zeros(heads * vdim, dtype=torch.bool)
    touched[[5, vdim + 3, vdim + 9]] = True
    for c in touched.nonzero().flatten().tolist():
        close(got[:, c], want[:, c], f"column {c}")
    assert torch.equal(got[:, ~touched], clean[:, ~touched])
    rows = lambda s: s.view(heads, dim, vdim).permute(0, 2, 1).reshape(heads * vdim, dim)
    assert torch.equal(rows(got_state)[~touched], rows(clean_state)[~touched])
    close(rows(got_state)[touched], rows(S.float())[touched], "state")


@pytest.mark.parametrize("lens", [[1] * 5, [3, 0, 1], [2, 40]])
@pytest.mark.parametrize("plain", [False, True])
@pytest.mark.parametrize("heads,kvh,dim,vdim", [(4, 2, 128, 128), (3, 1, 48, 4), (2, 2, 64, 64), (6, 2, 100, 68), (2, 1, 127, 132)])
def test_single_tokens_by_whole_lines(heads, kvh, dim, vdim, plain, lens):
    """A step said to bring one token a request, states in rows of whole 16 bytes: outputs and states against float64. What
    the step is said to bring decides the order of the sums only: requests that bring none or several are right too."""
    from hi_b200.kernels import ops

    n, g = sum(lens), torch.Generator().manual_seed(dim + vdim)
    rnd = lambda *s: torch.randn(*s, generator=g)
    q, k = (F.normalize(rnd(n, kvh, dim), dim=-1).reshape(n, -1) for _ in range(2))
    v, beta, decay = rnd(n, heads * vdim), torch.rand(n, heads, generator=g), torch.rand(n, heads * dim, generator=g)
    cu, slots = tables(lens)
    state = rnd(len(lens) + 2, heads * dim * vdim + 4)
    dev = state.to(DEV)
    o = ops.delta_recurrence(q.to(DEV), k.to(DEV), v.to(DEV), None if plain else beta.to(DEV), decay.to(DEV), dev, cu.to(DEV),
                             slots.to(DEV), heads, kvh, dim, vdim, single_tokens=True, plain=plain).cpu()
    dev = dev.cpu()
    for i, slot in enumerate(slots.tolist()):
        S = state[slot, : heads * dim * vdim].double().view(heads, dim, vdim)
        for t in range(int(cu[i]), int(cu[i + 1])):
            wide = lambda x: x[t].double().view(kvh, dim).repeat_interleave(heads // kvh, dim=0)
            S = S * decay[t].double().view(heads, dim, 1)
            vt = v[t].double().view(heads, vdim)
            u = vt if plain else beta[t].double()[:, None] * (vt - torch.einsum("hdv,hd->hv", S, wide(k)))
            S = S + wide(k)[:, :, None] * u[:, None, :]
            close(o[t], torch.einsum("hdv,hd->hv", S, wide(q)).reshape(-1), f"output {t}")
        close(dev[slot, : heads * dim * vdim], S.reshape(-1), f"state {slot}")
        assert torch.equal(dev[slot, heads * dim * vdim:], state[slot, heads * dim * vdim:])
    for slot in set(range(len(lens) + 2)) - set(slots.tolist()):
        assert torch.equal(dev[slot], state[slot])


# by shares (the first: of the scratch as it is) with blocks of 16 and of 32 columns, and in order, where most requests' first chunks
# fill the scratch: launches that hold different requests
@pytest.mark.parametrize("heads,dim,vdim,lens,scratch", [(64, 128, 8, [5, 2300, 600, 1, 33], 0), (3, 96, 80, [130, 1, 17, 260, 40], 1 << 20),
                                                         (16, 64, 128, [200, 0, 150, 40, 1], 5 << 20), (8, 33, 70, [20] * 30, 4 << 20),
                                                         (16, 128, 100, [100, 3, 40, 70], 1 << 19)])
@pytest.mark.parametrize("rule", ["delta", "plain", "mlstm"])
def test_steps_that_take_several_slices_of_scratch(rule, heads, dim, vdim, lens, scratch, monkeypatch):
    """More prepared chunks than the scratch holds: the states go from launch to launch, wherever a request's chunks are cut."""
    from hi_b200.kernels import ops

    n, g, cols = sum(lens), torch.Generator(device=DEV).manual_seed(3), vdim + (rule == "mlstm")
    if scratch:
        monkeypatch.setattr(ops, "CHUNKED_SCRATCH_BYTES", scratch)
    size = lambda *a: ops._chunked_scratch(*a, dim, cols, rule != "delta", "cpu").numel()
    assert size(n, len(lens), max(lens), heads) < (n // 16 + len(lens)) * heads * size(1, 1, 1, 1)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    cu, slots = tables(lens)
    kw = dict(longest=max(lens))
    monkeypatch.setattr(ops, "_chunked_recurrence", lambda *a, **k: True)
    if rule == "mlstm":
        proj = 0.5 * rnd(n, heads * (2 * dim + vdim))
        q, k, v = (t.reshape(n, heads, -1).double() for t in proj.split([heads * dim, heads * dim, heads * vdim], dim=1))
        v = torch.cat([v, torch.ones(n, heads, 1, dtype=torch.float64, device=DEV)], dim=2)
        keep, take = torch.rand(n, heads, device=DEV, generator=g), torch.rand(n, heads, device=DEV, generator=g)
        state = 0.3 * rnd(len(lens) + 2, ops.mlstm_state_floats(heads, dim, vdim))
        after = state.clone()
        o, nq = ops.mlstm_recurrence(proj, 0, heads * dim, 2 * heads * dim, dim ** -0.5, keep, take, after, cu.to(DEV), slots.to(DEV), heads,
                                     dim, vdim, **kw)
        o = torch.cat([o.view(n, heads, vdim), nq.view(n, heads, 1)], dim=2).reshape(n, -1)
        q, v, decay = q * dim ** -0.5, v * take.double()[:, :, None], keep.double()[:, :, None].expand(n, heads, dim)
        shape, order = (heads, cols, dim), lambda S: S.permute(0, 2, 1)
    else:
        q, k = (F.normalize(rnd(n, heads, dim), dim=-1) for _ in range(2))
        v, beta = rnd(n, heads, vdim), torch.rand(n, heads, device=DEV, generator=g)
        decay = torch.exp(-torch.exp(2.0 * rnd(n, heads, dim) - 2.0))
        state = rnd(len(lens) + 2, heads * dim * vdim)
        after = state.clone()
        o = ops.delta_recurrence(q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1), None if rule == "plain" else beta, decay.reshape(n, -1),
                                 after, cu.to(DEV), slots.to(DEV), heads, heads, dim, vdim, plain=rule == "plain", **kw)
        q, k, v, decay = q.double(), k.double(), v.double(), decay.double()
        shape, order = (heads, dim, cols), lambda S: S
    for s, slot in enumerate(slots.tolist()):
        if lens[s] == 0:
            assert torch.equal(after[slot], state[slot])
            continue
        S, want = order(state[slot, : heads * dim * cols].double().view(shape)), []
        for t in range(int(cu[s]), int(cu[s + 1])):
            S = S * decay[t][:, :, None]
            u = v[t] if rule != "delta" else beta[t].double()[:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            want.append(torch.einsum("hdv,hd->hv", S, q[t]).reshape(-1))
        close(o[int(cu[s]): int(cu[s + 1])], torch.stack(want), f"request {s}")
        close(order(after[slot, : heads * dim * cols].view(shape)), S, f"state {s}")
