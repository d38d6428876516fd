"""Decode attention whose splits meet inside a cluster of blocks, against the softmax in float64 and against the splits merged
by a kernel of their own: 2 to 8 splits, tokens that have fewer of them than the batch's longest, every page size."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nh,nkv,hd", [(40, 8, 128), (8, 2, 64), (3, 3, 128), (16, 1, 64)])
@pytest.mark.parametrize("lens,page,chunk,sink,splits", [([300, 1, 64, 128, 63], 16, 0, True, 2), ([900, 300, 512, 513], 128, 512, True, 2),
                                                         ([513, 2], 32, 0, False, 3), ([1000], 64, 0, False, 4), ([1100, 40, 257], 16, 0, True, 5),
                                                         ([1500, 1], 32, 0, False, 6), ([1791, 700, 256], 16, 0, True, 7), ([1900, 3, 257], 64, 0, True, 8),
                                                         # one split, and more than a cluster has: the same kernels either way
                                                         ([65, 1, 64, 128, 63], 16, 0, True, 1), ([129, 700, 64], 64, 128, False, 1), ([2100], 64, 0, False, 9)])
def test_splits_meet_in_a_cluster(nh, nkv, hd, lens, page, chunk, sink, splits, monkeypatch):
    from hi_b200.kernels import ops

    g = torch.Generator().manual_seed(sum(lens) + nh)
    n, pages = len(lens), sum(-(-k // page) for k in lens)
    q = torch.randn(n, nh, hd, generator=g).to(torch.bfloat16)
    kp, vp = (torch.randn(pages, nkv, page, hd, generator=g).to(torch.bfloat16) for _ in range(2))
    order, at = torch.randperm(pages, generator=g).to(torch.int32), 0
    table = torch.full((n, max(-(-k // page) for k in lens)), -1, dtype=torch.int32)
    for i, k in enumerate(lens):
        need = -(-k // page)
        table[i, :need] = order[at: at + need]
        at += need
    pos = torch.tensor([k - 1 for k in lens], dtype=torch.int32)
    args = [t.to(DEV) for t in (q, kp, vp, table, torch.arange(n, dtype=torch.int32), pos)]
    call = lambda: ops.decode_attention(*args, chunk, 0, hd ** -0.5, max(lens), sink=sink)
    # every number of splits from 1 to 9 runs for rows of either length, whatever the model of the time would choose
    longest = min(max(lens), chunk or max(lens))
    size = -(-(-(-longest // 64)) // splits) * 64
    assert -(-longest // size) == splits
    asked = []
    monkeypatch.setattr(ops, "_decode_splits", lambda *a: (asked.append(a), (size, splits))[1])
    before = ops.CALLS.get("attention_merge", 0)
    got = call()
    assert ops.CALLS.get("attention_merge", 0) - before == (splits > 8)
    assert asked == [(longest, n * nkv, hd, 0)]
    assert torch.equal(got, call())                        # the blocks of a cluster finish in any order: the sum has one
    monkeypatch.setattr(ops, "DECODE_CLUSTER", 1)
    apart = call()
    assert ops.CALLS.get("attention_merge", 0) - before == (1 < splits <= 8) + 3 * (splits > 8)
    for i, k in enumerate(lens):
        lo = (k - 1) // chunk * chunk if chunk else 0
        rows = lambda t: t[table[i, : -(-k // page)].long()].transpose(1, 2).reshape(-1, nkv, hd)[lo:k].double()
        ks, vs = (rows(t).repeat_interleave(nh // nkv, dim=1) for t in (kp, vp))
        scores = torch.einsum("hd,khd->hk", q[i].double(), ks) * hd ** -0.5
        top = scores.max(dim=1, keepdim=True).values
        e = torch.exp(scores - top)
        want = torch.einsum("hk,khd->hd", e, vs) / (e.sum(1, keepdim=True) + (torch.exp(-top) if sink else 0.0))
        # weights rounded to bfloat16 (2^-9 each, averaged over the keys) and the result rounded once more: 2^-8 of the largest
        err = float((got[i].cpu().double() - want).abs().max() / want.abs().max())
        assert err < 2 ** -7, (i, err)
    # the same sums in the same order: at most the last place of bfloat16 where a product was contracted differently
    assert float((got.float() - apart.float()).abs().max()) <= 2 ** -8 * float(apart.float().abs().max())


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("splits", [2, 5, 6, 8, 9])
def test_clusters_only_where_all_run_at_once(splits, hd, monkeypatch):
    from hi_b200.kernels import ops

    fit = ops._decode_clusters(0, hd, splits)
    assert (fit == 0) == (splits > 8) and fit * splits <= 148 * 8
    monkeypatch.setattr(ops, "_decode_splits", lambda *a: (64, splits))
    g = torch.Generator(device=DEV).manual_seed(splits)
    for n in (max(1, fit), fit + 1):
        q, kp, vp = (torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((n, 4, hd), (n * splits, 1, 64, hd), (n * splits, 1, 64, hd)))
        table = torch.arange(n * splits, dtype=torch.int32, device=DEV).view(n, splits)
        pos = torch.randint(0, 64 * splits, (n,), device=DEV, generator=g).to(torch.int32)
        call = lambda: ops.decode_attention(q, kp, vp, table, torch.arange(n, dtype=torch.int32, device=DEV), pos, 0, 0, hd ** -0.5, 64 * splits)
        before = ops.CALLS.get("attention_merge", 0)
        got = call()
        assert ops.CALLS.get("attention_merge", 0) - before == (n > fit)
        with monkeypatch.context() as m:
            m.setattr(ops, "DECODE_CLUSTER", 1)
            assert float((got.float() - call().float()).abs().max()) <= 2 ** -8 * float(got.float().abs().max())      # one bfloat16 place


# by a cluster, by the merge of several rounds' splits, of more than eight splits, by the cp.async kernel (rows of 192, a window, kept
# tokens, a cap, a bias and a learned sink), the sink of all of them
@pytest.mark.parametrize("nh,nkv,hd,lens,window,merged,more", [
    (8, 2, 128, [900, 1, 300], 0, False, {}), (8, 2, 64, [900, 1, 300], 0, False, {"sink": True}), (8, 8, 64, [600, 480] * 15, 0, True, {}),
    (4, 1, 64, [9000, 64], 0, True, {"sink": True}), (8, 4, 192, [300, 77, 1000], 0, True, {}), (8, 2, 64, [1500, 3], 1024, True, {}),
    (8, 2, 128, [1500, 3, 700], 512, True, {"keep": 100}), (6, 2, 64, [700, 20], 0, True, {"softcap": 5.0, "slopes": 1}),
    (6, 2, 128, [700, 20], 0, True, {"sink_values": 1})])
def test_tokens_decoded_where_they_lie_in_a_step(nh, nkv, hd, lens, window, merged, more, monkeypatch):
    from hi_b200.kernels import ops

    general = ops._decode_splits                            # these cuts, whatever the kernel's own model would choose
    monkeypatch.setattr(ops, "_decode_splits", lambda longest, groups, *a: general(longest, groups))

    g = torch.Generator(device=DEV).manual_seed(hd + len(lens))
    page, n = 64, len(lens)
    need = [-(-k // page) for k in lens]
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16)
    kp, vp = rnd(sum(need), nkv, page, hd), rnd(sum(need), nkv, page, hd)
    table, at = torch.zeros(n, max(need), dtype=torch.int32, device=DEV), 0
    for i, k in enumerate(need):
        table[i, :k] = torch.arange(at, at + k)
        at += k
    total = 3 * n + 5                                       # tokens of the step; every third or so is a decoded one
    rows = (torch.randperm(total, device=DEV, generator=g)[:n]).sort().values
    q, out = rnd(total, nh, hd), rnd(total, nh, hd)
    i32 = lambda: torch.zeros(total, dtype=torch.int32, device=DEV)
    seq, pos = i32(), i32()
    seq[rows] = torch.arange(n, dtype=torch.int32, device=DEV)
    pos[rows] = torch.tensor([k - 1 for k in lens], dtype=torch.int32, device=DEV)
    more = {k: torch.rand(nh, device=DEV, generator=g) if k in ("slopes", "sink_values") else v for k, v in more.items()}
    rest = (hd ** -0.5, max(lens))
    called = ops.CALLS.get("attention_merge", 0)
    want = ops.decode_attention(q[rows], kp, vp, table, seq[rows], pos[rows], 0, window, *rest, **more)
    assert ops.CALLS.get("attention_merge", 0) - called == merged
    before = out.clone()
    assert ops.decode_attention(q, kp, vp, table, seq, pos, 0, window, *rest, rows=rows, out=out, **more) is out
    assert torch.equal(out[rows], want)                     # the same kernels and cuts, other addresses
    others = torch.ones(total, dtype=torch.bool, device=DEV)
    others[rows] = False
    assert torch.equal(out[others], before[others])
    ops.check_tc_status()
    # rows that the step does not have are left out and found
    wrong, out = rows.clone(), before.clone()
    wrong[0], wrong[-1] = -1, total
    ops.decode_attention(q, kp, vp, table, seq, pos, 0, window, *rest, rows=wrong, out=out, **more)
    with pytest.raises(ops.KernelError, match="row outside the step"):
        ops.check_tc_status()
    ops.check_tc_status()
    assert torch.equal(out[rows[1:-1]], want[1:-1])
    others[rows[0]] = others[rows[-1]] = True
    assert torch.equal(out[others], before[others])


def test_an_output_is_given_with_its_rows():
    from hi_b200.kernels import ops

    q, pages = torch.zeros(2, 4, 64, dtype=torch.bfloat16, device=DEV), torch.zeros(2, 1, 64, 64, dtype=torch.bfloat16, device=DEV)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    rows = torch.tensor([1], device=DEV)
    for seq, pos, more in ((i32(0, 1), i32(3, 3), {"out": q.clone()}), (i32(0, 1), i32(3, 3), {"rows": rows}),
                           (i32(0), i32(3, 3), {"rows": rows, "out": q.clone()}), (i32(0, 1), i32(3), {"rows": rows, "out": q.clone()})):
        with pytest.raises(ops.KernelError):
            ops.decode_attention(q, pages, pages, i32(0, 1).view(2, 1), seq, pos, 0, 0, 0.125, 4, **more)
