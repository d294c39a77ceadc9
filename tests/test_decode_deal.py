"""How the one-launch decode step deals the blocks of keys to the CTAs, on the host: the function is the kernel's own."""
import ctypes
import os
import random

import numpy as np
import pytest

BLOCK, CTAS, EXTRA = 32, 148, 13


def deal(positions, heads, kv_heads, ctas=CTAS):
    from purhie_b200.csrc import build
    lib = ctypes.CDLL(os.path.join(build.build_dir(), build.library_file("layers")))
    pos = np.asarray(positions, dtype=np.int32)
    out = np.zeros((ctas * 8 + 8 * kv_heads * 8, 9), dtype=np.int32)
    n = lib.ph_decode_layers_deal(len(positions), heads, kv_heads, pos.ctypes.data_as(ctypes.c_void_p), ctas,
                                  out.ctypes.data_as(ctypes.c_void_p), len(out))
    assert 0 < n <= len(out)
    return out[:n]


def check(positions, heads, kv_heads, ctas=CTAS):
    """Every block of every (row, head) once, in order; a pair's pieces in consecutive CTAs, each of which knows how many there are; at
    most two pieces of a CTA that wait for a merge, and not of the same side."""
    pieces = deal(positions, heads, kv_heads, ctas)
    pairs, sides = {}, set()
    for cta, row, head, b0, n, blocks, parts, index, first in pieces.tolist():
        assert n > 0 and blocks == positions[row] // BLOCK + 1
        assert cta == first + index and 0 <= index < parts
        pairs.setdefault((row, head), []).append((index, b0, n, parts, blocks))
        if parts > 1:
            assert (cta, index == 0) not in sides
            sides.add((cta, index == 0))
    assert len(pairs) == len(positions) * kv_heads
    for held in pairs.values():
        held.sort()
        assert [h[0] for h in held] == list(range(held[0][3]))
        at = 0
        for _, b0, n, parts, blocks in held:
            assert b0 == at and parts == len(held)
            at += n
        assert at == held[0][4]
    cost = np.zeros(ctas)
    for p in pieces:
        cost[p[0]] += p[4] + EXTRA
    return cost.max()


@pytest.mark.parametrize("seed", range(40))
def test_every_block_is_dealt_once(seed):
    rng = random.Random(seed)
    for _ in range(25):
        rows, kv = rng.randint(1, 8), rng.choice([1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 40])
        longest = rng.choice([1, 40, 300, 2500, 40000, 200000])
        positions = [rng.randrange(longest) for _ in range(rows)]
        check(positions, kv * rng.randint(1, 8), kv, rng.choice([148, 148, 132, 64, 7, 1]))


@pytest.mark.parametrize("positions,heads,kv_heads,most", [
    ([32767] * 5, 16, 16, 1.10),                   # five long rows: whole CTAs leave the largest piece at 1.85 of the even share
    ([32767] + [255] * 7, 16, 16, 1.35),           # one long row beside short ones: 4.6
    ([32767] + [255] * 7, 32, 32, 1.35),           # more pairs than CTAs: a pair that is never cut is 4.2
    ([8191] * 7, 32, 8, 1.15),
    ([2047] * 8, 32, 32, 1.25),
])
def test_the_longest_share_is_near_the_even_one(positions, heads, kv_heads, most):
    blocks = [p // BLOCK + 1 for p in positions]
    even = kv_heads * sum(b + EXTRA for b in blocks) / CTAS + EXTRA
    assert check(positions, heads, kv_heads) <= most * even


def test_a_short_row_of_few_heads_is_not_cut_beyond_what_its_merge_costs():
    assert max(p[6] for p in deal([2047], 16, 2).tolist()) <= 20
    assert max(p[6] for p in deal([2047], 16, 8).tolist()) == 18
