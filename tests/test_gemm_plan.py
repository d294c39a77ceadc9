"""Into how many parts a product cuts K: the parts decide in which type a result is handed on and in which order it is added
up, so they do not follow from what tiles happen to be fast."""
import pytest

SMS = 148


def parts_of_k(M, N, K):
    """The rule, restated: units of a block of 64 of K on 128 x 256 tiles; 0.87 of one on pairs of SMs (256 x 256); six for an
    item's start and epilogue; 0.33 us to a unit where partial sums travel at 4 TB/s."""
    up = lambda a, b: -(-a // b)
    blocks, best = up(K, 64), None
    for rows, slots, unit in ((128, SMS, 1.0), (256, SMS // 2, 0.87)):
        if rows == 256 and (M <= 128 or N <= 128):
            continue
        for s in (1, 2, 3, 4, 6, 8):
            if s > 1 and blocks // s < 8:
                continue
            cost = up(up(M, rows) * up(N, 256) * s, slots) * (unit * blocks / s + 6.0) + (2.0 * s * M * N * 4 / 4e12 / 0.33e-6 if s > 1 else 0)
            if best is None or cost < best[0] - 1e-9:
                best = (cost, s)
    return best[1]


def plan(M, N, K, allow_split=True, fused=False):
    from purhie_b200 import native
    return native.answer(native.lib().qe_plan_gemm(M, N, K, SMS, int(allow_split), int(fused)))


# projections whose K was left whole (q and k rounded to bfloat16 in front of their norm) while their cut was left to the tiles
@pytest.mark.parametrize("N,K,first,last", [(4096, 1024, 128, 140), (3072, 1024, 167, 186), (4096, 1536, 187, 210), (2048, 1536, 374, 420),
                                            (5120, 1024, 128, 128)])
def test_projections_hand_float32_sums_to_their_norm(N, K, first, last):
    for M in (first, (first + last) // 2, last):
        assert plan(M, N, K)["splits"] > 1


@pytest.mark.parametrize("N,K", [(129, 1024), (1024, 2048), (1024, 3072), (3072, 2048), (4096, 1024), (4096, 4096), (4096, 12288), (6144, 4096),
                                 (2048, 8192), (6656, 2048), (520, 200)])
def test_the_parts_of_k_are_the_rules(N, K):
    for M in list(range(128, 700, 7)) + [1024, 1151, 1153, 1536, 2047, 2048]:
        p = plan(M, N, K)
        assert p["splits"] == parts_of_k(M, N, K) and not p["swapped"]
        assert p["block_n"] == 256 or not p["pair"]
        assert p["splits"] == 1 or p["block_n"] > 64
        assert plan(M, N, K, allow_split=False)["splits"] == plan(M, N, K, fused=True)["splits"] == 1
