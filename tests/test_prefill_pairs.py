"""The tcgen05 prefill attention of two query tiles a block: where pairs, tiles, steps of 16 keys and shares of the keys end."""
import random
import time

import pytest
import torch

from hi_b200.kernels import ops

DEV = "cuda:0"


def reference(q, k, v, starts, lens, chunk, window, scale, sinks):
    out, at = torch.zeros(q.shape, dtype=torch.float64), 0
    group = q.shape[1] // k[0].shape[1]
    for s, (c, n) in enumerate(zip(starts, lens)):
        pos, key = torch.arange(c, c + n).view(-1, 1), torch.arange(c + n).view(1, -1)
        hidden = key > pos
        if chunk:
            hidden |= key < pos // chunk * chunk
        if window:
            hidden |= key <= pos - window
        for h in range(q.shape[1]):
            kk, vv = (x[s][:, h // group].double() for x in (k, v))
            scores = (q[at: at + n, h].double() @ kk.t() * scale).masked_fill(hidden, float("-inf"))
            if sinks is not None:
                scores = torch.cat([scores, sinks[h].double().expand(n, 1)], dim=1)
                vv = torch.cat([vv, torch.zeros(1, vv.shape[1], dtype=torch.float64)])
            out[at: at + n, h] = torch.softmax(scores, 1) @ vv
        at += n
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd,page,chunk,window,lens,starts,sink", [
    (5, 1, 128, 64, 0, 0, [300, 128, 1, 129], [0, 37, 500, 127], False),        # odd groups: a pair of two tiles; single items
    (3, 3, 128, 16, 0, 0, [257, 1], [128, 3], True),                            # a group of one: pairs of tiles of one head
    (2, 1, 64, 64, 0, 0, [128], [0], False),                                    # one block
    (10, 2, 64, 32, 300, 0, [385, 140, 17], [250, 299, 300], False),            # chunks that start inside tiles and steps
    (4, 2, 128, 64, 0, 100, [260, 131], [700, 0], False),                       # windows: pages before them were given back
    (40, 8, 64, 128, 0, 0, [700, 400, 513, 2], [0, 260, 5, 900], False),        # more pairs than SMs: blocks take another
])
def test_pairs_of_query_tiles(nh, nkv, hd, page, chunk, window, lens, starts, sink):
    g = torch.Generator().manual_seed(nh * hd + page)
    total, S = [c + n for c, n in zip(starts, lens)], len(lens)
    k, v = ([torch.randn(t, nkv, hd, generator=g).bfloat16() for t in total] for _ in range(2))
    q = torch.randn(sum(lens), nh, hd, generator=g).bfloat16()
    need = [-(-t // page) for t in total]
    pages = torch.randperm(sum(need), generator=g).int()
    # whatever no token may read holds NaN: the rows behind a request's end, and page 0's stand-in for pages given back
    kp, vp = (torch.full((sum(need) + 1, nkv, page, hd), float("nan"), dtype=torch.bfloat16) for _ in range(2))
    table, at = torch.full((S, max(need)), -1, dtype=torch.int32), 0
    for s in range(S):
        first = starts[s] // chunk * chunk if chunk else max(0, starts[s] - window + 1) if window else 0
        for b in range(need[s]):
            slot = int(pages[at + b]) + 1
            here = slice(b * page, min((b + 1) * page, total[s]))
            kp[slot, :, : here.stop - here.start], vp[slot, :, : here.stop - here.start] = (x[s][here].transpose(0, 1) for x in (k, v))
            if (b + 1) * page > first:
                table[s, b] = slot
        at += need[s]
    cu = torch.tensor([0] + lens).cumsum(0).int()
    pos = torch.cat([torch.arange(c, c + n) for c, n in zip(starts, lens)]).int()
    sinks = torch.randn(nh, generator=g) if sink else None
    want = reference(q, k, v, starts, lens, chunk, window, hd ** -0.5, sinks)
    dev = lambda x: None if x is None else x.to(DEV)
    assert ops.prefill_pairs(hd)
    for splits in (1, 2, 5):
        got = ops.prefill_attention_tc(dev(q), dev(kp), dev(vp), dev(table), dev(cu), dev(pos), S, max(lens), chunk, window, hd ** -0.5,
                                       key_splits=splits, sink_values=dev(sinks))
        ops.check_tc_status()
        # P in bfloat16 (2^-9 of each weight, weights that sum to one) and the output's own rounding, on values of a few units
        err = float((got.double().cpu() - want).abs().max())
        assert err <= 2e-2, (splits, err)
        if 1 not in lens:
            continue
        out = torch.full_like(dev(q), 7.0)
        ops.prefill_attention_tc(dev(q), dev(kp), dev(vp), dev(table), dev(cu), dev(pos), S, max(lens), chunk, window, hd ** -0.5,
                                 key_splits=splits, sink_values=dev(sinks), skip_single=True, out=out)
        ops.check_tc_status()
        alone = int(cu[lens.index(1)])
        rest = [i for i in range(q.shape[0]) if i != alone]
        assert torch.equal(out[rest], got[rest])
        if splits == 1:
            assert bool((out[alone] == 7.0).all()), "a single token is left to the decode kernel"


@pytest.mark.parametrize("portions,nh,nkv,hd,chunk,window,least,want", [
    ([(0, 2048)], 40, 8, 128, 0, 0, 1, {1}), ([(7000, 128)], 40, 8, 128, 8192, 0, 1, {4, 5, 6, 7, 8}), ([(0, 128)], 8, 2, 64, 0, 0, 1, {1}),
    ([(0, 2048)], 40, 8, 128, 0, 0, 2, {2, 3, 4, 5, 6, 7, 8}), ([(9000, 150), (300, 700)], 40, 8, 128, 0, 0, 1, {2, 3, 4}),
    ([(100000, 128)], 16, 4, 128, 0, 64, 1, {1}), ([], 40, 8, 128, 0, 0, 1, {1}), ([(500, 128)], 8, 2, 128, 0, 0, 1, {1}),
    ([(20000, 4096)], 24, 24, 64, 0, 0, 1, {1}), ([(65000, 200)], 1, 1, 64, 0, 0, 1, {6, 7, 8})])
def test_shares_of_pairs(portions, nh, nkv, hd, chunk, window, least, want):
    """Prompts from the start, short launches and those that fill the GPU stay in one share; few long pairs are shared out."""
    rows = sum(n for _c, n in portions)
    assert ops.prefill_pair_shares(portions, nh, nkv, hd, chunk, window, rows, 148, least) in want


@pytest.mark.gpu
@pytest.mark.parametrize("capture", [False, True])
def test_single_tokens_decoded_aside(capture, monkeypatch):
    """Single tokens beside portions that leave SMs idle go on a second stream: the same rows as one after the other, call after call
    on memory that the calls before gave back, and in a captured step."""
    from hi_b200.parts import attention as part
    from hi_b200.parts.context import StepContext

    g = torch.Generator(device=DEV).manual_seed(3)
    nh, nkv, hd, page = 8, 2, 128, 64
    lens, starts = [300, 1, 130, 1, 1], [6600, 900, 0, 3, 2500]
    total = [c + n for c, n in zip(starts, lens)]
    need = [-(-t // page) for t in total]
    table, at = torch.zeros(len(lens), max(need), dtype=torch.int32, device=DEV), 0
    for s, k in enumerate(need):
        table[s, :k] = torch.arange(at, at + k)
        at += k
    kp, vp = (torch.randn(at, nkv, page, hd, device=DEV, generator=g).bfloat16() for _ in range(2))
    q = torch.randn(sum(lens), nh, hd, device=DEV, generator=g).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu = [0] + [sum(lens[: i + 1]) for i in range(len(lens))]
    singles = [i for i, n in enumerate(lens) if n == 1]
    ctx = StepContext(n_tokens=cu[-1], n_seqs=len(lens), tokens=i32([0] * cu[-1]),
                      positions=torch.cat([torch.arange(c, c + n) for c, n in zip(starts, lens)]).int().to(DEV),
                      seq_of_token=i32([s for s, n in enumerate(lens) for _ in range(n)]), cu_seqlens=i32(cu),
                      slots=i32(list(range(len(lens)))), start_pos=starts, n_new=lens, slot_ids=list(range(len(lens))), page_size=page,
                      max_context=max(total))
    ctx.decode_rows = torch.tensor([cu[i] for i in singles], dtype=torch.int64, device=DEV)
    ctx.decode_max_context = max(total[i] for i in singles)
    monkeypatch.setattr(ops, "prefill_pair_shares", lambda *a: 1)
    idle = ops.prefill_pair_idle_us(((6600, 300), (0, 130)), nh, nkv, hd, 0, 0, ops.sm_count(q.device))
    assert idle >= part.DECODE_ASIDE_IDLE_US
    call = lambda: part.attend_over_pages(q, kp, vp, table, ctx, nh, nkv, hd, 0, 0, hd ** -0.5)
    monkeypatch.setattr(part, "DECODE_ASIDE_KEYS", 0)       # the same cut either way
    with monkeypatch.context() as m:
        m.setattr(part, "DECODE_ASIDE_IDLE_US", 1e9)
        want = call()
    if capture:
        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = call()
        for _ in range(5):
            got.zero_()
            graph.replay()
            assert torch.equal(got, want)
    else:
        for _ in range(20):
            got = call()
            again = torch.full_like(got, 3.0)          # (may take memory that the call gave back)
            assert torch.equal(got, want) and float(again.float().mean()) == 3.0
            del got, again
    ops.check_tc_status()


@pytest.mark.parametrize("portions,nh,nkv,chunk,window,want", [
    ([(0, 160)], 40, 8, 0, 0, True), ([(0, 161), (0, 105)], 16, 4, 0, 0, True), ([(5, 315)], 16, 4, 8192, 4096, True), ([(0, 448)], 8, 8, 0, 0, True),
    ([(0, 128)], 40, 8, 0, 0, False), ([(0, 200)], 40, 8, 0, 0, False), ([(0, 449)], 8, 2, 0, 0, False), ([(0, 513)], 8, 2, 0, 0, False),
    ([(0, 300)], 40, 8, 0, 0, True), ([(0, 300), (0, 130)], 40, 8, 0, 0, False), ([(0, 300)], 8, 2, 256, 0, False), ([(0, 300)], 8, 2, 0, 100, False),
    ([], 8, 2, 0, 0, False), ([(400, 140), (0, 150)], 8, 2, 0, 0, False), ([(0, 300)], 8, 8, 0, 0, False), ([(0, 180)], 8, 8, 0, 0, True)])
def test_short_launches_that_go_one_query_tile_a_block(portions, nh, nkv, chunk, window, want):
    """One round of blocks whose last 128 keys are half empty: two tiles a block took 1.05 to 1.2 of the time there."""
    assert ops.prefill_one_tile(portions, nh, nkv, chunk, window) is want


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd,lens,sink", [(8, 2, 128, [160, 1, 131], False), (4, 2, 64, [300, 17], True)])
def test_one_query_tile_a_block_gives_the_same_rows(nh, nkv, hd, lens, sink, monkeypatch):
    from hi_b200.parts import attention as part
    from hi_b200.parts.context import StepContext

    g = torch.Generator(device=DEV).manual_seed(hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    need = -(-max(lens) // 64)
    kp, vp, q = rnd(len(lens) * need, nkv, 64, hd), rnd(len(lens) * need, nkv, 64, hd), rnd(sum(lens), nh, hd)
    table = torch.arange(len(lens) * need, dtype=torch.int32, device=DEV).view(len(lens), need)
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    ctx = StepContext(n_tokens=cu[-1], n_seqs=len(lens), tokens=i32([0] * cu[-1]), positions=torch.cat([torch.arange(n) for n in lens]).int().to(DEV),
                      seq_of_token=i32([s for s, n in enumerate(lens) for _ in range(n)]), cu_seqlens=i32(cu), slots=i32(list(range(len(lens)))),
                      start_pos=[0] * len(lens), n_new=lens, slot_ids=list(range(len(lens))), page_size=64, max_context=max(lens))
    ctx.decode_rows, ctx.decode_max_context = (torch.tensor([cu[lens.index(1)]], device=DEV), 1) if 1 in lens else (None, 0)
    sinks = torch.randn(nh, device=DEV, generator=g) if sink else None
    call = lambda: part.attend_over_pages(q, kp, vp, table, ctx, nh, nkv, hd, 0, 0, hd ** -0.5, sink_values=sinks)
    seen, real = [], ops.prefill_attention_tc
    monkeypatch.setattr(ops, "prefill_attention_tc", lambda *a, **k: (seen.append(k["one_tile"]), real(*a, **k))[1])
    one = call()
    monkeypatch.setattr(ops, "prefill_one_tile", lambda *a: False)
    two = call()
    ops.check_tc_status()
    assert seen == [True, False]
    rows = lambda t, s: t[table[s].long()].transpose(1, 2).reshape(-1, nkv, hd)[: lens[s]].cpu()
    want = reference(q.cpu(), [rows(kp, s) for s in range(len(lens))], [rows(vp, s) for s in range(len(lens))], [0] * len(lens), lens, 0, 0, hd ** -0.5,
                     None if sinks is None else sinks.cpu())
    for got in (one, two):      # as in the test of the pairs
        assert float((got.double().cpu() - want).abs().max()) <= 2e-2


def shares_in_plain_python(portions, nh, nkv, hd, chunk, window, rows, sms, least, most=8):
    """The model as it reads: runs of neighbouring pairs, and for every number of shares the longest block, the average SM and the turns."""
    runs, group = [], nh // nkv
    for cached, new in portions:
        items = -(-new // 128) * group
        pairs = -(-items // 2)
        n = min(8, pairs)
        for i in range(n):
            a, b = pairs * i // n, pairs * (i + 1) // n
            first, end = cached + 128 * ((a + b - 1) // group), min(cached + 128 * (min(a + b, items - 1) // group + 1), cached + new) - 1
            seen = max(first // chunk * chunk if chunk else 0, first - window + 1 if window else 0)
            runs.append((end // 128 - seen // 128 + 1, (b - a) * nkv))
    fixed, tile, merge, share, whole = (7.75, 1.515, 1.46, 0.6, 6.2) if hd <= 64 else (8.4, 1.73, 1.27, 0.63, 4.05)

    def cost(k):
        tiles = sorted(((-(-t // k) + 0.5, n * k) for t, n in runs), reverse=True)
        longest, before = max(tiles[0][0], sum(t * n for t, n in tiles) / sms), 0
        for t, n in tiles:
            before += n
            longest = max(longest, ((before - 1) // sms + 1) * t)
        return fixed + tile * longest + (merge + (share * k + whole) * rows * nh * hd / 1e6 if k > 1 else 0.0)

    if not runs:
        return 1, 0.0
    idle = tile * (max(t for t, _n in runs) - sum(t * n for t, n in runs) / sms)
    best = min(range(least, most + 1), key=cost)
    return (best if least > 1 or cost(best) < min(0.93 * cost(1), cost(1) - 8.0) else 1,
            max(0.0, idle) if tile * max(t for t, _n in runs) >= 80.0 else 0.0)


def test_the_plan_of_a_launch_costs_the_host_little():
    """The search in the library gives what the model says, and a step whose portions are new to it does not wait for it: in Python it took
    60 us for one portion and 289 for eight, as long as the kernel that it plans for."""
    rng = random.Random(7)
    steps = []
    for _ in range(300):
        nh, nkv = rng.choice([(40, 8), (16, 4), (8, 2), (24, 24), (5, 1), (3, 3)])
        portions = tuple((rng.choice([0, rng.randint(0, 70000)]), rng.randint(1, rng.choice([2, 200, 4000]))) for _ in range(rng.choice([0, 1, 2, 8])))
        chunk, window = rng.choice([(0, 0), (8192, 0), (300, 0), (0, 1024), (512, 100)])
        steps.append((portions, nh, nkv, rng.choice([64, 128]), chunk, window, sum(n for _c, n in portions), rng.choice([148, 132, 1]), rng.choice([1, 1, 2, 5])))
    ops.lib()
    took = [0.0, 0.0]
    for step in steps:
        t0 = time.perf_counter()
        got = ops.prefill_pair_shares(list(step[0]), *step[1:]), ops.prefill_pair_idle_us(*step[:6], step[7])
        t1 = time.perf_counter()
        assert got == shares_in_plain_python(*step), step
        took = [took[0] + t1 - t0, took[1] + time.perf_counter() - t1]
    assert took[0] < 0.5 * took[1], took
    with pytest.raises(ops.KernelError, match="no shares"):
        ops.prefill_pair_shares([(0, 128)], 5, 2, 128, 0, 0, 128, 148)
    with pytest.raises(ops.KernelError, match="no time"):
        ops.prefill_pair_idle_us(((0, -1),), 4, 2, 128, 0, 0, 148)
