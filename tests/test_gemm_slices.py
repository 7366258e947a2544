"""Into how many slices along K a product of many tokens is cut, and which of them are taken whole: by the cost of tiles of 256 columns."""
import math
import random

import pytest

SMS, LEAST, OVERHEAD, NARROW = 148, 16, 12, 2 << 20      # multiprocessors, k-blocks of a slice and a tile's overhead, bytes of planes that may be cut finer


def _lib():
    from kestrel_llm_b200.csrc import ops
    return ops.library()


def _cost(T, N, K, s):
    """(cost in k-blocks of a pair's time, rounds of tiles) of s slices; None where they are not whole or too short."""
    kb, pairs = -(-K // 64), SMS // 2
    per = -(-kb // s)
    if s > 1 and (per < LEAST or -(-kb // per) != s):
        return None
    rounds = -(-(-(-N // 256) * -(-T // 256) * s) // pairs)
    return rounds * (OVERHEAD + per) + max(0, 8 * T * N * (s - 1) - (64 << 20)) // 2100000, rounds


def _slices(T, N, K):
    return min((s for s in range(1, 9) if _cost(T, N, K, s)), key=lambda s: (_cost(T, N, K, s)[0], s))


def _sizes():
    rng = random.Random(3)

    def spread(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    return [(spread(129, 8192), 8 * spread(2, 16384), 8 * spread(8, 2048)) for _ in range(3000)]


def test_a_product_has_no_fewer_slices_than_whole_tiles_give_it():
    """A sum's distance from float64 grows with the length of its slices: tiles narrower than 256 columns do not take slices away."""
    lib = _lib()
    for T, N, K in _sizes() + [(512, 6144, 4096), (449, 6144, 4096), (1024, 6144, 4096), (2048, 3088, 2048), (1777, 3216, 2048), (1000, 32, 2048)]:
        want, got = _slices(T, N, K), lib.kestrel_gemm_tc_splits(T, N, K)
        assert got == want or (got > want and 4 * T * N * got <= NARROW), (T, N, K, want, got)


@pytest.mark.parametrize("N,K,taken", [(6144, 4096, [(144, 0), (300, 0), (448, 0), (449, 0), (512, 0), (513, 1), (768, 1), (769, 0), (1000, 0), (1024, 0), (1025, 1),
                                                      (1536, 1), (1537, 1), (1792, 1), (2048, 1), (3072, 1)]),
                                       (3072, 2048, [(144, 0), (512, 0), (768, 0), (769, 1), (1024, 1), (1536, 1), (1537, 0), (2048, 0), (2304, 0), (2305, 1), (3072, 1)])])
def test_which_query_key_value_products_are_taken_whole(N, K, taken):
    """With the work of the kernel that prepares attention in the epilogue: uncut, or in three rounds of tiles and more where cutting gains
    less than a tenth."""
    lib = _lib()
    for T, want in taken:
        assert lib.kestrel_gemm_tc_qkv_whole(T, N, K) == want, T
    for T, _, _ in _sizes()[:500]:
        S = _slices(T, N, K)
        whole, rounds = _cost(T, N, K, 1)
        assert lib.kestrel_gemm_tc_qkv_whole(T, N, K) == (S == 1 or (rounds >= 3 and whole * 10 <= _cost(T, N, K, S)[0] * 11)), T


def test_the_tile_taken_costs_least_with_those_slices():
    """Of tiles of 128 to 256 columns: a k-block costs as much as its columns, or as 236 where the operands' way in sets the pace."""
    lib = _lib()
    chosen = set()
    for T, N, K in _sizes() + [(1024, 3072, 2048), (300, 4096, 4096), (2048, 4096, 4096)]:
        S = lib.kestrel_gemm_tc_splits(T, N, K)
        per, planes = -(-(-(-K // 64)) // S), 256 * (max(0, 8 * T * N * (S - 1) - (64 << 20)) // 2100000)

        def cost(columns):
            rounds = -(-(-(-N // 256) * -(-T // columns) * S) // (SMS // 2))
            return rounds * ((128 + columns // 2) * OVERHEAD + per * max(columns, 236)) + planes
        got = lib.kestrel_gemm_tc_pair_columns(T, N, K, S)
        assert got == min(range(256, 127, -16), key=lambda c: (cost(c), -c)), (T, N, K, S)
        chosen.add(got)
    assert len(chosen) >= 6 and 256 in chosen


@pytest.mark.gpu
@pytest.mark.parametrize("T,N,K", [(512, 6144, 4096), (2048, 3088, 2048), (1000, 6144, 4096), (300, 4096, 4096)])
def test_sums_are_as_close_to_float64_as_in_those_slices(T, N, K):
    """Products of bfloat16 numbers are exact in float32, so the distance is that of the sums alone; of as many terms it differs by less than
    a hundredth from draw to draw of the operands."""
    import torch
    from kestrel_llm_b200.csrc import ops
    off = []
    for seed, S in ((0, None), (0, _slices(T, N, K)), (1, _slices(T, N, K))):
        gen = torch.Generator("cuda").manual_seed(seed)
        x, w = torch.randn((T, K), device="cuda", generator=gen).bfloat16(), (torch.randn((N, K), device="cuda", generator=gen) * K ** -0.5).bfloat16()
        y = ops.Partials(ops.gemm_tc(x, w, splits=S), None).reduce(torch.float32)
        want = x.double() @ w.double().T
        off.append(float((y.double() - want).norm() / want.norm()))
    ops.raise_on_kernel_error()
    assert off[0] <= 1.02 * max(off[1:]), off
