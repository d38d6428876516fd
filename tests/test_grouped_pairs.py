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
