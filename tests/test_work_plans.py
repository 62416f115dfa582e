"""How calls are cut up for the device, by size: host arithmetic, no GPU."""
import ctypes as C

import pytest

SMS = 148


def attention_plan(dim, q_heads, kv_heads, tokens, sms=SMS):
    """(ranges, parts of a job, whole jobs) of a batch of sequences."""
    from turboquant_mlx_core_b200 import _lib
    ranges, parts, whole = C.c_int(), C.c_int(), C.c_int()
    assert _lib.load().tq_kv_attention_plan(dim, q_heads, kv_heads, len(tokens), (C.c_int * len(tokens))(*tokens), sms, C.byref(ranges), C.byref(parts),
                                            C.byref(whole)) == 0
    return ranges.value, parts.value, whole.value


def _tiles(out, rows):
    return -(-out // 128) * -(-rows // 256)


# q / k / v and gate / up of hidden sizes that a decoder has: with few rows all of a group's CTAs run side by side.  (More than the SMs cost
# 20 to 35 %.)
GROUPS = [(1024, (1024, 256, 256), 1024), (1024, (1024, 1024, 1024), 512), (1024, (4096, 4096), 256), (1280, (1280, 256, 256), 1024),
          (1536, (1536, 1536, 1536), 256), (1792, (1792, 256, 256), 512), (2048, (2048, 256, 256), 256), (2048, (2048, 512, 512), 256),
          (2048, (2048, 2048), 256), (2048, (3072, 768, 768), 256), (2560, (2560, 512, 512), 256), (3072, (1024, 1024, 1024), 256)]


@pytest.mark.parametrize("cols,outs,most", GROUPS)
def test_groups_fit_the_device(cols, outs, most):
    from turboquant_mlx_core_b200 import _lib
    lib = _lib.load()
    for rows in (9, 16, 32, 64, 128, 256, 300, 512, 1024):
        if rows <= most:
            assert sum(_tiles(o, rows) * lib.tq_linear_k_splits(o, cols, rows, 1, SMS) for o in outs) <= SMS, rows


def test_splits_of_k():
    """Eight blocks of 64 columns a split at least, no more CTAs than SMs, at least one split."""
    from turboquant_mlx_core_b200 import _lib
    lib = _lib.load()
    for planes in (1, 2):
        for cols in (64, 512, 768, 960, 1024, 1088, 4096, 18944, 28672):
            for out in (1, 512, 3584, 8192, 37888, 151936):
                for rows in (9, 256, 257, 2048):
                    s = lib.tq_linear_k_splits(out, cols, rows, planes, SMS)
                    assert s >= 1 and (s == 1 or (cols // 64 * planes // s >= 8 and s * _tiles(out, rows) <= SMS))
    assert lib.tq_linear_k_splits(8192, 512, 128, 1, SMS) == 1     # (the sums would outweigh what the CTAs gain)
    assert lib.tq_linear_k_splits(512, 100, 9, 1, SMS) == -1 and lib.tq_linear_k_splits(512, 128, 0, 1, SMS) == -1


# Where cutting every job into as many parts was slower than whole jobs or equal shares (us: without, with parts).
NOT_IN_PARTS = [
    (64, 8, 8, [552, 609, 168, 504], 7.8, 8.3), (128, 40, 8, [552, 609, 168, 504], 8.2, 8.6), (64, 8, 1, [552, 609, 168, 504], 7.8, 8.2),
    (32, 8, 1, [1000] * 32, 7.4, 7.8), (32, 28, 4, [1000] * 7 + [40], 7.4, 7.8), (64, 4, 2, [1000] * 32, 10.3, 10.7), (64, 8, 1, [3000, 40], 11.6, 12.6),
    (32, 32, 8, [9892, 3906, 2504, 7455, 11953, 11778, 11340, 12986], 25.5, 29.9), (128, 8, 1, [126] * 63 + [4000], 15.9, 16.8),
    (256, 28, 4, [8000] * 8, 59.1, 61.1),
]


@pytest.mark.parametrize("case", NOT_IN_PARTS, ids=[f"{len(c[3])}x{max(c[3])}_q{c[1]}_kv{c[2]}_d{c[0]}" for c in NOT_IN_PARTS])
def test_attention_is_not_cut_where_that_costs(case):
    dim, q_heads, kv_heads, tokens, _, _ = case
    assert attention_plan(dim, q_heads, kv_heads, tokens)[1] == 0


def test_equal_shares_where_whole_jobs_are_slower():
    assert attention_plan(256, 28, 4, [4000] * 31 + [40]) == (148, 0, 0)     # 101.4 us, whole jobs 106.2


def test_attention_in_parts():
    """Few long jobs; a part has a tile of every job at least, and no more ranges than a device has places for."""
    for dim, q_heads, kv_heads, tokens in ((128, 28, 4, [4096]), (128, 28, 4, [32768]), (128, 40, 8, [8192]), (128, 28, 4, [1024] * 8), (64, 8, 8, [4096] * 16),
                                           (256, 8, 2, [2048] * 4), (32, 8, 1, [16384])):
        ranges, parts, whole = attention_plan(dim, q_heads, kv_heads, tokens)
        assert parts >= 2 and whole == 0 and ranges == parts * len(tokens) * kv_heads * -(-q_heads // kv_heads // 8)
        assert ranges <= (SMS if dim == 256 else 2 * SMS)
    assert attention_plan(128, 8, 2, [5000, 100])[1] == 7           # 7 tiles of 16 tokens
    assert attention_plan(128, 8, 1, [5000] * 8 + [16])[1] == 0


def test_attention_plans_of_drawn_batches():
    """Every range has work to do or there are as few as jobs; equal shares never more than two a multiprocessor."""
    import random
    rng = random.Random(5)
    for _ in range(3000):
        dim, kv_heads, n = rng.choice([32, 64, 128, 256]), rng.choice([1, 2, 4, 8]), rng.choice([1, 1, 2, 3, 8, 33, 200])
        q_heads = kv_heads * rng.choice([1, 4, 5, 7, 8, 9])
        tokens = [int(10 ** rng.uniform(0, 5)) for _ in range(n)]
        sms = rng.choice([1, 20, 132, 148])
        ranges, parts, whole = attention_plan(dim, q_heads, kv_heads, tokens, sms)
        jobs, tiles = n * kv_heads * -(-q_heads // kv_heads // 8), [-(-t // 16) for t in tokens]
        assert 1 <= ranges <= min(320, 2 * sms) and not (parts and whole)
        if parts:
            assert ranges == jobs * parts and 2 <= parts <= min(tiles)
        elif whole:
            assert ranges <= jobs
        else:
            assert ranges <= max(1, sum(tiles) * jobs // n)


def test_attention_plan_refuses():
    from turboquant_mlx_core_b200 import _lib
    r = [C.c_int() for _ in range(3)]
    refs = [C.byref(x) for x in r]
    one, none = (C.c_int * 1)(5), (C.c_int * 1)(0)
    plan = _lib.load().tq_kv_attention_plan
    assert plan(96, 4, 4, 1, one, SMS, *refs) == -1 and plan(128, 5, 4, 1, one, SMS, *refs) == -1 and plan(128, 4, 4, 0, one, SMS, *refs) == -1
    assert plan(128, 4, 4, 1, none, SMS, *refs) == -1 and plan(128, 4, 4, 1, None, SMS, *refs) == -1 and plan(128, 4, 4, 1, one, SMS, *refs) == 0
