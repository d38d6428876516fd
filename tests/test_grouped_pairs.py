"""Grouped expert products by pairs of blocks (256 weight rows a tile): where tiles, halves of tokens, k blocks and pieces end."""
import pytest
import torch

from hi_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("experts,hidden,inter,counts", [
    (2, 72, 136, [511, 1]),                      # ragged features, k blocks and tokens; an odd token alone; nothing for a block's half
    (3, 1024, 264, [769, 0, 0]),                 # an expert with everything: tiles of equal shares, the last features in the even block
    (2, 200, 4096, [193, 387]),                  # a long k: the last round is cut
    (1, 2048, 520, [300]),                       # one expert
    (4, 512, 1024, [127, 129, 385, 383]),        # either side of a slot and of a tile
])
def test_pairs_of_blocks(experts, hidden, inter, counts):
    g = torch.Generator(device=DEV).manual_seed(inter)
    rows = sum(counts)
    assert rows >= 256 * experts
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x = rnd(rows, hidden).bfloat16()
    wg, wu, wd = ((rnd(*s) * s[-1] ** -0.5).bfloat16() for s in ((experts, inter, hidden), (experts, inter, hidden), (experts, hidden, inter)))
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])[torch.randperm(rows)].to(DEV)
    scores = torch.rand(rows, device=DEV, generator=g)
    plan = ops.moe_plan(ids.view(-1, 1).contiguous(), experts)
    act = ops.moe_gate_up_tc(x, plan, 1, wg, wu, scores)
    relu = ops.moe_up_relu2_tc(x, plan, 1, wu)
    down = ops.moe_down_tc(act, wd, plan)
    again = ops.moe_down_tc(act, wd, plan)
    ops.check_tc_status()
    order = plan.sorted_entry.long()
    xs, of, s = x.double()[order], ids.long()[order], scores.double()[order][:, None]
    gate, up = (torch.einsum("rk,rfk->rf", xs, w.double()[of]) for w in (wg, wu))
    # bfloat16 results of float32 sums of k products of order one: 2^-9 of the value, and the sums' own error (k 2^-24 at the most)
    close = lambda got, want: float((got.double() - want).abs().max()) <= 2 ** -8 * float(want.abs().max())
    assert close(act, torch.nn.functional.silu(s * gate) * (s * up))
    assert close(relu, torch.relu(up) ** 2)
    want = torch.einsum("rk,rfk->rf", act.double(), wd.double()[of])
    assert float((down.double() - want).abs().max()) <= inter * 2 ** -23 * float(want.abs().max())
    assert torch.equal(down, again)              # whichever piece comes last


def gate_up_tile(counts, inter, hidden, paired, sms=148):
    """The most tokens of a tile of gate and up, as dual_tokens chooses on the device: fewest bytes into an SM over the rounds."""
    few, many = sum(-(-c // 192) for c in counts), sum(-(-c // 128) for c in counts)
    if all(c <= 128 * -(-c // 192) for c in counts):
        return 192
    units, features, stages = (sms // 2, -(-inter // 256), -(-hidden // 64)) if paired else (sms, -(-inter // 128), -(-hidden // 64))
    return 128 if -(-many * features // units) * 48 * stages < -(-few * features // units) * (56 * stages + 480) else 192


@pytest.mark.parametrize("limit", [0.0, 1.5])
@pytest.mark.parametrize("experts,hidden,inter,counts,paired,tile", [
    (1, 2048, 8192, [576], True, 192),           # three tiles of 192: both slots of tensor memory are one tile's, in both blocks
    (2, 1000, 3560, [570, 381], True, 192),      # ragged ones: 190 and 191 tokens, the last features in the even block
    (2, 512, 1032, [571, 381], True, 128),
    (4, 2048, 2432, [130, 261, 250, 10], False, 192),       # one block a tile, either side
    (4, 512, 1024, [130, 261, 250, 10], False, 128),
    (3, 200, 136, [140, 0, 150], False, 128),
])
def test_gate_and_up_by_tiles_of_either_length(experts, hidden, inter, counts, paired, tile, limit):
    rows = sum(counts)
    assert rows > 256 and (rows >= 256 * experts) == paired and ops.sm_count(DEV) == 148
    assert gate_up_tile(counts, inter, hidden, paired) == tile
    g = torch.Generator(device=DEV).manual_seed(inter + rows)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g)
    x = rnd(rows, hidden).bfloat16()
    wg, wu = ((rnd(experts, inter, hidden) * hidden ** -0.5).bfloat16() for _ in range(2))
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])[torch.randperm(rows)].to(DEV)
    scores = torch.rand(rows, device=DEV, generator=g)
    plan = ops.moe_plan(ids.view(-1, 1).contiguous(), experts)
    act = ops.moe_gate_up_tc(x, plan, 1, wg, wu, scores, limit)
    ops.check_tc_status()
    order = plan.sorted_entry.long()
    xs, of, s = x.double()[order], ids.long()[order], scores.double()[order][:, None]
    gate, up = torch.zeros(rows, inter, device=DEV, dtype=torch.float64), torch.zeros(rows, inter, device=DEV, dtype=torch.float64)
    for e in range(experts):
        gate[of == e], up[of == e] = (s[of == e] * (xs[of == e] @ w[e].double().t()) for w in (wg, wu))
    want = gate.clamp(max=limit) * torch.sigmoid(1.702 * gate.clamp(max=limit)) * (up.clamp(-limit, limit) + 1) if limit else \
        torch.nn.functional.silu(gate) * up
    # a bfloat16 result of float32 sums of products of order one: 2^-9 of the value, and the sums' own error
    assert float((act.double() - want).abs().max()) <= 2 ** -8 * float(want.abs().max())


def test_as_many_rows_as_the_other_products_take():
    """8.4 million rows are 43,751 tiles of 192 tokens, which all three products take, and more than 65,535 of 128."""
    rows, hidden = 8_400_000, 8
    g = torch.Generator(device=DEV).manual_seed(1)
    x, scores = torch.randn(rows, hidden, device=DEV, generator=g).bfloat16(), torch.rand(rows, device=DEV, generator=g)
    wg, wu = (torch.randn(1, hidden, hidden, device=DEV, generator=g).bfloat16() for _ in range(2))
    entry = torch.arange(rows, dtype=torch.int32, device=DEV)
    plan = ops.MoePlan(torch.tensor([0, rows], dtype=torch.int32, device=DEV), entry, entry, torch.tensor([1, 0], dtype=torch.int32, device=DEV))
    act = ops.moe_gate_up_tc(x, plan, 1, wg, wu, scores)
    ops.check_tc_status()
    gate, up = (scores[:, None] * (x.float() @ w[0].float().t()) for w in (wg, wu))
    want = torch.nn.functional.silu(gate) * up
    # one rounding to bfloat16 on sums of eight products in float32
    assert bool(((act.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-4).all())
