"""Rules by which the host chooses a kernel's shape, for GPUs of a given number of SMs (CPU, no compute)."""
import ctypes
import heapq
import random

from conftest import pkg


def test_ranks_by_1024_threads_from_a_number_of_pairs_that_depends_on_the_waves():
    f = pkg("_lib").load().b200_moe_rank_threads
    assert [f(n, e, 148) for e in (1, 128, 148) for n in (0, 8191, 8192)] == [256, 256, 1024] * 3
    assert [f(n, e, 148) for e in (149, 256, 1024) for n in (8192, 16383, 16384)] == [256, 256, 1024] * 3
    assert f(8192, 149, 160) == 1024 and f(1, 0, 148) < 0


def test_row_tiles_of_dense_products():
    """Fewest waves of CTAs, then least data; a narrower tile that would need one wave more has to win by more than the estimate errs."""
    f = pkg("_lib").load().b200_dense_gemm_row_tile
    assert [f(m, 2048, 148) for m in (1300, 1500, 1777, 2048)] == [160, 192, 224, 256]
    assert f(4096, 5120, 148) == 256 and f(2246, 9216, 148) == 256 and f(1648, 12288, 148) == 256
    assert all(f(m, n, 148) % 32 == 0 and 32 <= f(m, n, 148) <= 256 for m in range(257, 4097, 37) for n in (100, 512, 5120, 10240))
    assert f(0, 2048, 148) < 0


def prefill_form(tokens, first, hq, hkv, chunk=0, sms=148):
    short = ctypes.c_int(-1)
    pairs = pkg("_lib").load().b200_paged_attn_prefill_pairs(tokens, first, hq, hkv, chunk, sms, ctypes.byref(short))
    return pairs, short.value


def walk_end(row_tiles, pairs, hkv, qt, first, tokens, chunk, sms):
    """When the last CTA of the grid ends if every SM takes the next one, late rows first: key tiles at 3 for one tile of rows and 4 for
    two, 12 for what is not the walk."""
    free, t, end = [0] * sms, row_tiles, 0
    for c in range(row_tiles - pairs):
        tiles = 2 if c < pairs else 1
        t -= tiles
        last = first + min((t + tiles) * qt, tokens) - 1
        lo = (first + t * qt) // chunk * chunk if chunk else 0
        length = (last // 128 - lo // 128 + 1) * (tiles + 2) + 12
        for _ in range(hkv):
            start = heapq.heappop(free)
            heapq.heappush(free, start + length)
            end = max(end, start + length)
    assert t == 0
    return end


def test_prompt_attention_takes_two_tiles_per_cta_where_that_ends_sooner():
    assert prefill_form(500, 333, 32, 4) == (0, 1)       # a tile per SM
    assert prefill_form(600, 0, 32, 4) == (0, 1)         # 152 tiles, single ones end sooner
    assert prefill_form(17, 3055, 32, 4) == (0, 1) and prefill_form(17, 3056, 32, 4) == (0, 0)  # 3072 keys and one more
    assert prefill_form(17, 9000, 32, 4, chunk=2048) == (0, 1)
    assert prefill_form(2048, 0, 32, 4) == (64, 0)
    assert prefill_form(1500, 14001, 32, 4) == (37, 0)   # 94 tiles: a wave of pairs, and one of single tiles
    assert prefill_form(1208, 5000, 32, 4) == (37, 0)    # 76 tiles
    assert prefill_form(0, 0, 32, 4)[0] < 0 and prefill_form(1, 0, 33, 4)[0] < 0
    rng, seen = random.Random(5), set()
    for _ in range(400):
        hq, hkv = rng.choice(((32, 4), (64, 4), (32, 8), (8, 8), (40, 8), (24, 8), (128, 1), (16, 2)))
        tokens, chunk = rng.randint(1, 4096), rng.choice((0, 0, 128, 500, 2048))
        first = rng.randint(0, 3 * tokens) if rng.random() < 0.7 else 0
        qt = 128 // (hq // hkv)
        tiles = -(-tokens // qt)
        pairs, _ = prefill_form(tokens, first, hq, hkv, chunk)
        assert 0 <= pairs <= tiles // 2
        if tiles * hkv <= 148:
            assert pairs == 0
        elif tiles * hkv <= 3 * 148 and (chunk or first <= tokens):
            none, every = (walk_end(tiles, p, hkv, qt, first, tokens, chunk, 148) for p in (0, tiles // 2))
            assert pairs == (tiles // 2 if every < none else 0)
            seen.add(pairs > 0)
    assert seen == {True, False}
