"""The decode attention by TMA: what its forms are compiled to, how they are cut, and the results at the cuts."""
import os
import re
import subprocess

import pytest
import torch

from hi_b200.kernels import build, ops

DEV = "cuda:0"


def test_the_fused_form_keeps_its_registers(tmp_path):
    """Its blocks an SM leave it the registers that it needs: held to the other forms' it spilled up to 224 bytes a thread."""
    source = os.path.join(build.CSRC, "attention_decode_tma.cu")
    out = subprocess.run([build._nvcc(), *build.ARCH_FLAGS, *build.NVCC_FLAGS, "-Xptxas", "-v", "-I", build.CSRC, "-c", source, "-o",
                          str(tmp_path / "x.o")], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, check=True).stdout
    spills = {name: int(n) for name, n in re.findall(r"Function properties for (\S+)\s+\d+ bytes stack frame, (\d+) bytes spill stores", out)}
    fused = {name: n for name, n in spills.items() if "attn_decode_tma_kernel" in name and "MergeE1E" in name}
    assert len(fused) == 2 and not any(fused.values()), spills


@pytest.mark.parametrize("hd,resident", [(64, 444), (128, 296)])
def test_the_fused_form_is_cut_for_its_own_merge_and_blocks(hd, resident):
    for groups in (1, 2, 8, 40, 100, 148, 149, 200, 222, 223, 256):
        for tiles in (1, 2, 3, 4, 7, 16, 33, 125, 1024, 4096):
            size, splits = ops._fused_splits(tiles, groups, hd)
            assert size % 64 == 0 and (splits - 1) * size < 64 * tiles <= splits * size and splits <= 48
            assert splits == 1 or size >= 128
            assert splits * groups <= resident or (splits <= 4 and 2 * groups > resident)
    want = {64: {(63, 64): {4, 5, 6}, (1, 256): {1}, (5, 256): {1}}, 128: {(128, 64): {4}, (32, 256): {1}, (1024, 32): {8, 9}, (128, 16): range(13, 19)}}
    for (tiles, groups), splits in want[hd].items():
        assert ops._fused_splits(tiles, groups, hd)[1] in splits, (tiles, groups)


@pytest.mark.gpu
@pytest.mark.parametrize("nh,nkv,hd", [(6, 2, 64), (16, 1, 128)])
@pytest.mark.parametrize("size", [64, 192, 256, 448])           # one tile a split; as many as are in flight; one more; the ring goes round
def test_fused_decode_at_the_ends_of_its_ring(nh, nkv, hd, size, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(size + hd)
    lens = [1, 64, 65, 193, 448, 449, 1000]
    need = [-(-k // 64) for k in lens]
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    kp, vp, qkv = rnd(sum(need), nkv, 64, hd), rnd(sum(need), nkv, 64, hd), rnd(len(lens), (nh + 2 * nkv) * hd)
    table, at = torch.full((len(lens), max(need)), -1, dtype=torch.int32, device=DEV), 0
    for i, k in enumerate(need):
        table[i, :k] = torch.arange(at, at + k)
        at += k
    pos = torch.tensor([k - 1 for k in lens], dtype=torch.int32, device=DEV)
    seq = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    monkeypatch.setattr(ops, "_fused_splits", lambda *a: (size, -(-max(lens) // size)))
    k1, v1 = kp.clone(), vp.clone()
    got = ops.decode_attention_fused(qkv, nh, nkv, hd, pos, None, False, False, 1e-6, None, seq, table, k1, v1, 0, 0, hd ** -0.5, max(lens))
    ops.check_tc_status()
    q, k_new, v_new = (x.view(len(lens), -1, hd) for x in qkv.split([nh * hd, nkv * hd, nkv * hd], dim=1))
    for i, k in enumerate(lens):
        rows = lambda t, new: torch.cat([t[table[i, : need[i]].long()].transpose(1, 2).reshape(-1, nkv, hd)[: k - 1], new[i: i + 1]]).double() \
            .repeat_interleave(nh // nkv, dim=1)
        p = torch.softmax(torch.einsum("hd,khd->hk", q[i].double(), rows(kp, k_new)) * hd ** -0.5, dim=1)
        want = torch.einsum("hk,khd->hd", p, rows(vp, v_new))
        # weights and the result in bfloat16, 2^-9 each, of the largest value
        assert float((got[i].double() - want).abs().max()) <= 2 ** -7 * float(want.abs().max()), (i, k)


@pytest.mark.gpu
@pytest.mark.parametrize("n,nh,nkv,longest,size", [
    (25, 24, 24, 128, 128), (64, 20, 10, 65, 128), (40, 24, 24, 64, 64),         # 600 to 960 blocks of one or two tiles: no warp for the loads
    (31, 24, 24, 140, 192), (50, 30, 15, 320, 320), (56, 24, 24, 300, 320),      # of three to five in a round less: places are given back
    (38, 16, 16, 300, 128), (47, 24, 24, 321, 384), (13, 24, 24, 300, 128)])     # several short splits a token; with the warp again
def test_rows_of_64_in_launches_of_many_blocks(n, nh, nkv, longest, size, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(n + longest)
    lens = [max(1, longest - 7 * i % longest) for i in range(n)]
    need = -(-longest // 32)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    kp, vp, q = rnd(n * need, nkv, 32, 64), rnd(n * need, nkv, 32, 64), rnd(n, nh, 64)
    table = torch.randperm(n * need, device=DEV, generator=g).int().view(n, need)
    pos = torch.tensor([k - 1 for k in lens], dtype=torch.int32, device=DEV)
    for i, k in enumerate(lens):                                # pages that a token does not reach are given back
        table[i, -(-k // 32):] = -1
    monkeypatch.setattr(ops, "_decode_splits", lambda *a: (size, -(-longest // size)))
    got = ops.decode_attention(q, kp, vp, table, torch.arange(n, dtype=torch.int32, device=DEV), pos, 0, 0, 0.125, longest)
    ops.check_tc_status()
    for i, k in enumerate(lens):
        rows = lambda t: t[table[i, : -(-k // 32)].long()].transpose(1, 2).reshape(-1, nkv, 64)[:k].double().repeat_interleave(nh // nkv, dim=1)
        p = torch.softmax(torch.einsum("hd,khd->hk", q[i].double(), rows(kp)) * 0.125, dim=1)
        want = torch.einsum("hk,khd->hd", p, rows(vp))
        # weights and the result in bfloat16, 2^-9 each, of the largest value
        assert float((got[i].double() - want).abs().max()) <= 2 ** -7 * float(want.abs().max()), (i, k)


def test_a_cut_is_searched_for_once_in_64_tokens(monkeypatch):
    monkeypatch.setattr(ops, "_decode_clusters", lambda *a: 50)
    ops._splits_of_tiles.cache_clear()
    for hd in (0, 64, 128):
        cuts = {ops._decode_splits(longest, 24, hd, 99) for longest in range(961, 1025)}
        assert len(cuts) == 1 and ops._decode_splits(1025, 24, hd, 99)[0] * ops._decode_splits(1025, 24, hd, 99)[1] >= 1025
    assert ops._splits_of_tiles.cache_info().misses == 8           # (rows of 128 ask the general rule too)
    ops._splits_of_tiles.cache_clear()


@pytest.mark.parametrize("hd,groups,tiles,splits", [(64, 96, 189, {6}), (64, 512, 16, {1}), (64, 8, 125, range(8, 25)), (64, 720, 2, {1})])
def test_rows_of_64_are_cut_for_one_round(hd, groups, tiles, splits, monkeypatch):
    fit = {2: 296, 3: 187, 4: 142, 5: 112, 6: 93, 7: 78, 8: 71}
    monkeypatch.setattr(ops, "_decode_clusters", lambda device, hd, real: fit[real])
    ops._splits_of_tiles.cache_clear()
    size, real = ops._decode_splits(64 * tiles, groups, hd, 99)
    ops._splits_of_tiles.cache_clear()
    assert real in splits and size % 64 == 0 and (real - 1) * size < 64 * tiles <= real * size


@pytest.mark.gpu
@pytest.mark.parametrize("longest,most,splits,size", [(10752, 2048, 6, 1792), (4097, 2048, 3, 1408), (2048, 2048, 1, 2048), (1000, 100, 8, 128), (130, 64, 3, 64)])
def test_no_split_is_longer_than_asked(longest, most, splits, size, monkeypatch):
    monkeypatch.setattr(ops, "_decode_splits", lambda keys, *a: (-(-keys // 64) * 64, 1))
    g = torch.Generator(device=DEV).manual_seed(longest)
    pages = -(-longest // 64)
    q, kp, vp = (torch.randn(*s, device=DEV, generator=g).bfloat16() for s in ((1, 4, 64), (pages, 2, 64, 64), (pages, 2, 64, 64)))
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    args = (q, kp, vp, torch.arange(pages, dtype=torch.int32, device=DEV).view(1, -1), i32(0), i32(longest - 1), 0, 0, 0.125, longest)
    acc, ml = ops.decode_attention(*args, parts=True, most_keys=most)
    assert acc.shape == (1, 4, splits, 64)
    for s in range(splits):                                     # every split its own run of keys: the sums of the weights by it
        keys = kp.transpose(1, 2).reshape(-1, 2, 64)[:longest][s * size:(s + 1) * size].double().repeat_interleave(2, dim=1)
        want = torch.logsumexp(torch.einsum("hd,khd->hk", q[0].double(), keys) * 0.125, dim=1)
        got = ml[0, :, s, 0].double() + ml[0, :, s, 1].double().log()
        assert float((got - want).abs().max()) <= 1e-4         # float32 sums of up to 2,048 terms
    whole = ops.decode_attention(*args)
    assert float((ops.decode_attention(*args, most_keys=most).float() - whole.float()).abs().max()) <= 2 ** -7 * float(whole.abs().max())
    ops.check_tc_status()


@pytest.mark.gpu
@pytest.mark.parametrize("hd", [64, 128])
def test_no_tokens_to_decode(hd):
    e = lambda *s, dtype=torch.bfloat16: torch.empty(*s, dtype=dtype, device=DEV)
    pages, none, table = torch.zeros(2, 2, 64, hd, dtype=torch.bfloat16, device=DEV), e(0, dtype=torch.int32), torch.zeros(1, 1, dtype=torch.int32, device=DEV)
    with pytest.raises(ops.KernelError, match="bad argument"):
        ops.decode_attention(e(0, 4, hd), pages, pages, e(0, 1, dtype=torch.int32), none, none, 0, 0, 0.125, 100)
    with pytest.raises(ops.KernelError, match="bad argument"):
        ops.decode_attention_fused(e(0, 8 * hd), 4, 2, hd, none, None, False, False, 1e-6, None, none, e(0, 1, dtype=torch.int32), pages, pages, 0, 0, 0.125, 100)
    q, out = torch.ones(3, 4, hd, dtype=torch.bfloat16, device=DEV), torch.full((3, 4, hd), 7.0, dtype=torch.bfloat16, device=DEV)
    three = torch.zeros(3, dtype=torch.int32, device=DEV)
    assert ops.decode_attention(q, pages, pages, table, three, three, 0, 0, 0.125, 100, rows=e(0, dtype=torch.int64), out=out) is out
    assert bool((out == 7.0).all())
