"""Float32 attention of portions on the tensor cores against softmax attention in float64: portions around the tiles of 64
rows and 32 keys, one-token requests beside them, every mask and score option, values that are not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# largest error over largest output: the weights' exponents carry up to |score| 2^-24 (scores up to about 10), the exponential
# and the sums of weights and values a few roundings of 6e-8 each
TOL = 3e-6


def setup(nh, nkv, hd, page, portions, seed=0):
    g = torch.Generator().manual_seed(seed)
    n = sum(m for m, _c in portions)
    need = [-(-(m + c) // page) for m, c in portions]
    pages = sum(need) + 1
    order = torch.randperm(pages, generator=g)[: sum(need)].to(torch.int32)
    table = torch.full((len(portions), max(need) + 1), -1, dtype=torch.int32)
    at = 0
    for s, k in enumerate(need):
        table[s, :k] = order[at: at + k]
        at += k
    q = torch.randn(n, nh, hd, generator=g)
    k, v = (torch.randn(pages, nkv, page, hd, generator=g) for _ in range(2))
    pos = torch.cat([torch.arange(c, c + m) for m, c in portions]).to(torch.int32)
    cu = torch.tensor([0] + list(torch.tensor([m for m, _c in portions]).cumsum(0)), dtype=torch.int32)
    return q, k, v, table, cu, pos


def reference(q, k, v, table, portions, chunk, window, keep, scale, softcap=0.0, slopes=None, sink=False, sink_values=None):
    n, nh, hd = q.shape
    nkv, page = k.shape[1], k.shape[2]
    out, at = torch.zeros(n, nh, hd, dtype=torch.float64), 0
    for s, (m, c) in enumerate(portions):
        ids = table[s, : -(-(m + c) // page)].long()
        p, j = torch.arange(c, c + m).view(-1, 1), torch.arange(m + c).view(1, -1)
        lo = torch.zeros_like(p)
        if chunk:
            lo = p // chunk * chunk
        if window:
            lo = torch.maximum(lo, p - window + 1)
        seen = (j <= p) & ((j >= lo) | (j < keep)) & (ids[j // page] >= 0)
        for h in range(nh):
            rows = lambda t: t[ids.clamp_min(0), h // (nh // nkv)].reshape(-1, hd)[: m + c].double()
            x = q[at: at + m, h].double() @ rows(k).t() * scale
            if softcap:
                x = softcap * torch.tanh(x / softcap)
            if slopes is not None:
                x = x - slopes[h].double() * (p - j)
            x = x.masked_fill(~seen, float("-inf"))
            if sink:
                x = torch.cat([x, torch.full((m, 1), 0.0 if sink_values is None else float(sink_values[h]), dtype=torch.float64)], 1)
            w = torch.softmax(x, dim=1)[:, : m + c]
            vv = torch.where(seen.any(0).view(-1, 1), rows(v), torch.zeros((), dtype=torch.float64))
            out[at: at + m, h] = w @ vv
        at += m
    return out


def run(case, portions, chunk=0, window=0, keep=0, **kw):
    from hi_b200.kernels import ops

    q, k, v, table, cu, pos = case
    dev = lambda t: t.to(DEV)
    kw = {n: dev(x) if torch.is_tensor(x) else x for n, x in kw.items()}
    o = ops.portion_attention(dev(q), dev(k), dev(v), dev(table), dev(cu), dev(pos), [m for m, _c in portions], chunk, window,
                              q.shape[2] ** -0.5, max(m + c for m, c in portions), keep=keep, **kw)
    assert o is not None
    return o.cpu()


def close(got, want):
    assert float((got.double() - want).abs().max() / want.abs().max()) <= TOL


@pytest.mark.parametrize("nh,nkv,hd", [(8, 2, 128), (2, 2, 16), (6, 1, 32), (5, 5, 48), (40, 8, 64), (4, 2, 80), (3, 1, 96),
                                       (2, 1, 112), (16, 1, 192)])
@pytest.mark.parametrize("portions", [[(2, 0)], [(64, 0), (1, 40), (65, 31)], [(33, 300), (1, 0), (130, 0)]])
def test_sizes(nh, nkv, hd, portions):
    page = 16 if hd % 3 else 24
    case = setup(nh, nkv, hd, page, portions)
    close(run(case, portions), reference(*case[:4], portions, 0, 0, 0, hd ** -0.5))


@pytest.mark.parametrize("chunk,window,keep", [(100, 0, 0), (0, 50, 0), (0, 40, 37), (128, 70, 0), (0, 1, 3)])
@pytest.mark.parametrize("options", [{}, {"softcap": 3.0, "sink": True}, {"slopes": True, "sink_values": True}])
def test_masks_and_scores(chunk, window, keep, options):
    portions = [(90, 210), (1, 77), (3, 0), (17, 120)]
    case = setup(4, 2, 64, 8, portions, seed=1)
    kw = {"softcap": options.get("softcap", 0.0), "sink": options.get("sink", False),
          "slopes": torch.rand(4) * 0.1 if options.get("slopes") else None,
          "sink_values": torch.randn(4) if options.get("sink_values") else None}
    got = run(case, portions, chunk, window, keep, **kw)
    close(got, reference(*case[:4], portions, chunk, window, keep, 0.125, **dict(kw, sink=kw["sink"] or kw["sink_values"] is not None)))


def test_shared_keys_holes_and_what_is_not_finite(monkeypatch):
    from hi_b200.kernels import ops

    portions = [(70, 500)]
    case = setup(4, 2, 128, 16, portions, seed=2)
    case[3][0, 7] = -1                                    # a page that is gone
    want = reference(*case[:4], portions, 0, 0, 0, 128 ** -0.5)
    for splits in (1, 3, 18):
        monkeypatch.setattr(ops, "portion_attention_splits", lambda blocks, keys: splits)
        close(run(case, portions), want)
    q, k, v, table, cu, pos = case
    at = 540                                              # the key of the 41st new token
    v[table[0, at // 16].long(), 0, at % 16, 3] = float("inf")
    got = run(case, portions)
    assert bool(torch.isinf(got[40:, :2, 3]).all())
    other = torch.ones_like(got, dtype=torch.bool)
    other[40:, :2, 3] = False
    assert float((got[other].double() - want[other]).abs().max() / want.abs().max()) <= TOL


def test_the_ends_of_the_range():
    """Finite numbers above bfloat16's largest (3.39e38) and infinite keys and queries: hidden ones change nothing for the
    rows that may not read them, a score of minus infinity weighs nothing, and a query reaches its own row only."""
    top = 3.4e38
    portions = [(70, 100)]
    q, k, v, table, cu, pos = setup(4, 2, 64, 16, portions, seed=5)
    args = (table, portions, 0, 0, 0, 0.125)
    at = 140                                              # the key of the 41st new token, hidden from the forty before it
    page, row = table[0, at // 16].long(), at % 16

    vt = v.clone()
    vt[page, 0, row, 3], vt[page, 1, row, 7] = top, -top
    got, want = run((q, k, vt, table, cu, pos), portions), reference(q, k, vt, *args)
    read = torch.zeros_like(got, dtype=torch.bool)
    read[40:, :2, 3] = read[40:, 2:, 7] = True
    assert float((got[read].double() - want[read]).abs().max()) <= TOL * top
    close(got[~read], want[~read])

    signs = torch.where(q[:, :2, 5].abs() > 0.02, q[:, :2, 5].sign(), torch.zeros(()))
    for big in (top, float("inf")):                       # the key outweighs everything or weighs nothing, as the query's sign says
        kt = k.clone()
        kt[page, 0, row, 5] = big
        got = run((q, kt, v, table, cu, pos), portions)
        plain = reference(q, k, v, *args)
        close(got[:40], plain[:40])
        close(got[:, 2:], plain[:, 2:])
        kt[page, 0, row, 5] = 1e30                        # (finite in float64 and in the reference's softmax)
        want = reference(q, kt, v, *args)
        nothing, all_of_it = torch.zeros(70, 4, dtype=torch.bool), torch.zeros(70, 4, dtype=torch.bool)
        nothing[40:, :2], all_of_it[40:, :2] = signs[40:] < 0, signs[40:] > 0
        assert bool(nothing.any()) and bool(all_of_it.any())
        close(got[nothing], want[nothing])
        if big == top:
            close(got[all_of_it], want[all_of_it])
        else:
            assert not bool(torch.isfinite(got[all_of_it]).any())

    qt = q.clone()
    qt[12, 1, 9] = float("inf")
    got, want = run((qt, k, v, table, cu, pos), portions), reference(q, k, v, *args)
    other = torch.ones(70, 4, dtype=torch.bool)
    other[12, 1] = False
    close(got[other], want[other])
    assert not bool(torch.isfinite(got[12, 1]).any())


@pytest.mark.parametrize("hd", [64, 128, 192])
@pytest.mark.parametrize("lens", [[1 + 128, 40], [31, 129 + 64], [97 + 128, 3], [33 + 256, 200]])
def test_tiles_with_few_tokens_in_the_bfloat16_kernel(hd, lens):
    """The tcgen05 kernel's warps without a token: the portion before gives what it gives alone, whatever the rows of the
    next request hold (here NaN), and the last rows of a ragged tile are right (bfloat16 weights and outputs: 2^-8 each)."""
    from hi_b200.kernels import ops

    portions = [(lens[0], 150), (lens[1], 70)]
    q, k, v, table, cu, pos = setup(4, 2, hd, 64, portions, seed=3)
    q, k, v = (t.to(torch.bfloat16) for t in (q, k, v))
    want = reference(q, k, v, table, portions, 0, 0, 0, hd ** -0.5)[: lens[0]]
    call = lambda qq: ops.prefill_attention_tc(qq.to(DEV), k.to(DEV), v.to(DEV), table.to(DEV), cu.to(DEV), pos.to(DEV), 2,
                                               max(lens), 0, 0, hd ** -0.5).cpu()[: lens[0]]
    got = call(q)
    assert float((got.double() - want).abs().max() / want.abs().max()) <= 2e-2
    q[lens[0]:] *= 100.0                                  # nor do the first one's last bits depend on them
    assert torch.equal(call(q), got)
    q[lens[0]:] = float("nan")
    assert torch.equal(call(q), got)
    ops.check_tc_status()


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,hd,splits", [(1, 16, 1), (7, 64, 2), (9, 128, 8), (40, 128, 9), (33, 192, 33), (5, 80, 70), (3, 1024, 5)])
def test_merge(rows, hd, splits, dt):
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(hd + splits)
    acc, ml = torch.randn(rows, splits, hd, generator=g), torch.randn(rows, splits, 2, generator=g) * 3
    ml[:, :, 1] = ml[:, :, 1].abs() + 0.1
    ml[0, (splits + 1) // 2:, 0] = float("-inf")          # splits beyond a token's range: never written
    acc[0, (splits + 1) // 2:] = float("nan")
    sinks = torch.randn(1, generator=g)
    acc_d, ml_d, sinks_d = acc.to(DEV), ml.to(DEV), sinks.to(DEV)
    for sink in (0, 1):
        out = torch.empty(rows, hd, dtype=dt, device=DEV)
        code = ops.lib().hb_attention_merge(acc_d.data_ptr(), ml_d.data_ptr(), out.data_ptr(),
                                            0 if dt == torch.float32 else 1, rows, hd, splits, sink, 1, sinks_d.data_ptr() if sink else None,
                                            torch.cuda.current_stream().cuda_stream)
        assert code == 0
        m = ml[:, :, 0].double()
        w = torch.exp(m - m.max(1, keepdim=True).values.clamp_min(-1e30))
        den = (w * ml[:, :, 1].double()).sum(1)
        if sink:
            den = torch.where(den > 0, den + torch.exp(sinks.double() - m.max(1).values), den)
        want = torch.where(w[:, :, None] > 0, w[:, :, None] * acc.double(), 0.0).sum(1) / den.clamp_min(1e-300)[:, None]
        err = float((out.cpu().double() - want).abs().max() / want.abs().max())
        assert err <= (2e-6 if dt == torch.float32 else 4e-3), err
