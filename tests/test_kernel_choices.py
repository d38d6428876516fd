"""Decisions that the Python side takes for the kernels, as plain functions of sizes and operands. No GPU."""
import pytest
import torch

from hi_b200.kernels import ops


def test_key_shares_of_the_tensor_core_prefill_attention():
    """Keys are shared among blocks only where the launch would leave most of the GPU waiting:
    few blocks, each with a long run of key tiles."""
    sms, places = 148, 296
    for blocks, tiles in ((40, 1017), (80, 1017), (160, 1020), (320, 1016), (300, 1000), (40, 600)):
        k = ops.prefill_key_splits(blocks, tiles, sms)
        assert 2 <= k <= 8 and tiles // k >= ops.PREFILL_SPLIT_MIN_SHARE, (blocks, tiles, k)
        fill = lambda n: (blocks * n / places) / -(-blocks * n // places)
        assert fill(k) > fill(1) and fill(k) >= max(fill(n) for n in range(1, 9) if tiles // n >= 128) - 0.05
    # launches of more than 1.25 rounds, short runs of keys, or nothing to do: one block each
    for blocks, tiles in ((1280, 992), (640, 500), (371, 2000), (160, 258), (40, 511), (0, 1000), (296, 1000)):
        assert ops.prefill_key_splits(blocks, tiles, sms) == 1, (blocks, tiles)
    # a smaller GPU has fewer places: the same launch is then more than its rounds' worth
    assert ops.prefill_key_splits(160, 1020, 40) == 1


def test_key_shares_of_any_mix_of_portions():
    """Few blocks with long runs of keys share them, chunked and windowed layers too; prompts from the start, launches that
    fill the GPU and nothing to do keep one block per query tile and head."""
    shares = lambda portions, nh=40, hd=128, chunk=0, window=0: ops.prefill_shares(portions, nh, hd, chunk, window,
                                                                                  sum(n for _c, n in portions), 148)
    assert shares([(7000, 128)]) > 1 and shares([(7000, 128)], chunk=8192) > 1 and shares([(100000, 128)], window=4096) > 1
    assert shares([(8190, 128)], chunk=8192) > 1                     # the tile reaches back over the chunk's end
    assert shares([(8192, 128)], chunk=8192) == 1 and shares([(9000, 128)], window=64) == 1
    assert shares([(9000, 150), (300, 700)]) > 1
    for portions in ([], [(0, 2048)], [(0, 128)], [(0, 512), (0, 1)], [(20000, 4096)], [(3000, 1024)]):
        assert shares(portions) == 1, portions
    for hd in (64, 128, 192):
        assert 1 <= shares([(50000, 1)], nh=1, hd=hd) <= 8


@pytest.mark.parametrize("heads,dim,vdim,lens,rule,faster", [
    (16, 128, 128, [48], "delta", True), (16, 128, 128, [24], "delta", False), (16, 128, 128, [512], "mlstm", True),
    (32, 64, 128, [8] * 64, "delta", False), (32, 64, 128, [449] + [1] * 63, "plain", False), (16, 16, 16, [512], "mlstm", True),
    (64, 64, 64, [128] * 8, "delta", False), (16, 128, 128, [16] * 64, "plain", True), (4, 64, 64, [24] * 32, "mlstm", False),
    (16, 129, 128, [2048], "delta", False), (16, 128, 128, [1] * 256, "mlstm", False), (16, 64, 64, [2048], "delta", True),
    # where chunks are prepared once a head, whatever its columns (us one by one / by chunks: 44 / 70, 175 / 208, 33 / 20, 397 / 289, 125 / 94)
    (32, 128, 16, [108] * 9, "delta", False), (20, 96, 32, [100] * 40, "delta", False), (10, 64, 80, [40] * 13, "mlstm", True),
    (40, 64, 80, [351] * 14, "plain", True), (16, 64, 128, [46] * 48, "plain", True)])
def test_recurrences_by_chunks_where_that_was_faster(heads, dim, vdim, lens, rule, faster):
    """Measured both ways (the rule before counted tokens and requests only and was up to 3.2 times slower)."""
    cols = vdim + (rule == "mlstm")
    assert ops._chunked_recurrence(sum(lens), len(lens), dim, rule, heads, cols, max(lens)) == faster


@pytest.mark.parametrize("nh,nkv,hd,portions,pays", [
    (16, 16, 128, [(100, 2)] + [(3400, 1)] * 31, False), (16, 4, 128, [(100, 2)] + [(3400, 1)] * 31, True),
    (24, 24, 64, [(100, 2)] + [(3400, 1)] * 31, False), (24, 24, 64, [(100, 2)] + [(760, 1)] * 63, True),
    (16, 16, 128, [(0, 64)] + [(760, 1)] * 63, False), (16, 16, 128, [(100, 2)] + [(250, 1)] * 31, True),
    (16, 16, 128, [(500, 300)] + [(3400, 1)] * 31, True), (8, 8, 64, [(500, 8), (3000, 1)], True), (40, 8, 128, [(0, 2048)], True),
    (4, 4, 192, [(0, 600)], True), (16, 16, 128, [(100, 2)], True)])
def test_float32_portions_by_tiles_where_that_was_faster(nh, nkv, hd, portions, pays):
    """Measured both ways, single tokens behind long contexts above all."""
    assert ops.portion_attention_pays(portions, nh, nkv, hd, 0, 0) == pays
    assert ops.portion_attention_pays(portions, nh, nkv, hd, 0, 128)        # a window leaves a few tiles a token


def test_products_of_a_few_rows_leave_foreign_operands_to_the_library(monkeypatch):
    """What is not on x's GPU, or x not on the current one, or wants gradients never reaches the kernel as a pointer."""
    class OnGpu(torch.Tensor):                # a host tensor that says it is on a GPU: no pointer of it may be used
        where = 0
        is_cuda = property(lambda self: True)
        device = property(lambda self: torch.device("cuda", self.where))

    def on(t, where=0):
        t = t.as_subclass(OnGpu)
        t.where = where
        return t

    monkeypatch.setattr(ops, "lib", lambda: pytest.fail("the kernel library was called"))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    bf16 = torch.bfloat16
    x, w, b = torch.zeros(2, 16, dtype=bf16), torch.zeros(32, 16, dtype=bf16), torch.zeros(32, dtype=bf16)
    assert ops.skinny_linear(on(x), w, bf16) is None
    assert ops.skinny_linear(on(x), on(w), bf16, b) is None
    assert ops.skinny_linear(on(x), on(w, 1), bf16) is None
    assert ops.skinny_linear(on(x, 1), on(w, 1), bf16, on(b, 1)) is None
    assert ops.skinny_linear(on(x), on(w).requires_grad_(), bf16) is None
    with torch.autograd.forward_ad.dual_level():
        assert ops.skinny_linear(on(x), on(w), bf16) is None
    with pytest.raises(ops.KernelError):
        ops.skinny_linear(x, w, bf16)
