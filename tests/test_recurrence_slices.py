"""How a step's chunks go through the recurrences' scratch, launch after launch, by the functions the launches use and without a GPU:
every chunk of every request once and in order, no two in one place, and requests side by side where the chain bounds the step."""
import ctypes
import random

import pytest

from hi_b200.kernels import ops

MB = 1 << 20


def launches(lens, heads, dim, cols, plain, most, longest=0):
    """Shares, units a launch, and [(request, chunk, count, unit)] of every launch in turn."""
    lib, n, s = ops.lib(), sum(lens), len(lens)
    call = lib.hb_recurrence_chunked_slices
    call.restype = None
    cu = (ctypes.c_int * (s + 1))(*[sum(lens[:i]) for i in range(s + 1)])
    out = (ctypes.c_int * 5)()
    step = (n, s, longest, heads, dim, cols, int(plain), ctypes.c_longlong(most))
    call(*step, None, 0, 0, 0, out)
    shares, units, got = out[0], out[1], []
    for share in range(shares):
        for unit0 in range(0, n // (16 * shares) + s, units):
            spans = []
            for r in range(s):
                call(*step, cu, r, share, unit0, out)
                if out[3] > 0:
                    spans.append((r, out[2], out[3], out[4]))
            got.append(spans)
    floats = lib.hb_recurrence_chunked_scratch_floats(*step)
    image = lib.hb_recurrence_chunked_scratch_floats(1, 1, 1, 1, dim, cols, int(plain), ctypes.c_longlong(1))      # of one chunk and head
    assert floats == units * heads * image and (4 * floats <= most or units == 1)
    return shares, units, got


def test_every_chunk_once_and_in_order():
    rng = random.Random(5)
    for _ in range(400):
        s = rng.choice([1, 2, 3, 7, 40])
        lens = [rng.choice([0, 1, 15, 16, 17, 33, rng.randint(1, 900)]) for _ in range(s)]
        if sum(lens) == 0:
            continue
        heads, dim, cols = rng.choice([1, 8, 64]), rng.choice([1, 32, 33, 64, 96, 128]), rng.choice([1, 16, 64, 129])
        _shares, units, got = launches(lens, heads, dim, cols, rng.random() < 0.5, int(MB * 2 ** rng.uniform(-6, 7)),
                                       rng.choice([0, max(lens), 10 ** 6]))
        done = [0] * s
        for spans in got:
            taken = set()
            for r, chunk, count, unit in spans:
                assert chunk == done[r]                     # the state goes from a launch to the next
                done[r] += count
                places = set(range(unit, unit + count))
                assert not places & taken and 0 <= unit and unit + count <= units
                taken |= places
        assert done == [-(-n // 16) for n in lens]


@pytest.mark.parametrize("lens,heads", [([4096] * 2, 16), ([2048] * 4, 16), ([1024] * 8, 16), ([2048] * 4, 8), ([2048] * 4, 32), ([4096, 1, 1, 1, 4000], 16),
                                        ([4000, 4000] + [1] * 120, 16)])
def test_long_requests_stay_side_by_side(lens, heads):
    """The chunks in turn are those of the longest request, not of one request after another."""
    shares, _units, got = launches(lens, heads, 128, 128, False, ops.CHUNKED_SCRATCH_BYTES, max(lens))
    assert sum(max(count for _r, _c, count, _u in spans) for spans in got if spans) <= -(-max(lens) // 16) + shares


def test_short_requests_go_in_order():
    """Where a slice's blocks fill the SMs anyway no request is cut more often than the scratch asks."""
    shares, units, got = launches([100] * 64, 64, 128, 128, False, ops.CHUNKED_SCRATCH_BYTES, 100)
    assert shares == 1 and len(got) == -(-(64 * 100 // 16 + 64) // units)
