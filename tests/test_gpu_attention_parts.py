"""Decode attention by the way its work is cut: every job (sequence, KV head, 8 query heads) in as many parts as the others - parts of a single tile,
of unequal tiles, lengths that end inside a tile, ranges that begin inside one, jobs of other lengths beside each other, one part an SM and
more of them than SMs - and equal shares of more ranges than SMs, whole jobs.  Each case says which way it is meant to take, and asserts it.
Against the oracle; tolerance as for the other splits of the work (test_gpu_attention_ranges).  The logs of the softmax
denominators: a score s is off by 2^-12 |s| for the query's rounding, of at most 8 that count, and the sum averages that: 4e-3."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.golden.make_golden import kv_inputs
from tests.test_work_plans import attention_plan

pytestmark = pytest.mark.gpu

TOL = 2.1e-3
LSE_TOL = 4e-3
CASES = [
    # tokens of each sequence, query heads, KV heads, head size, first token; on 148 SMs: ranges, parts of a job, whole jobs
    ([1024], 28, 4, 128, 0, (32, 8, 0)),
    ([1000, 1017], 8, 2, 128, 0, (32, 8, 0)),
    ([2100], 10, 1, 128, 37, (24, 12, 0)),              # two groups of query heads
    ([4099], 8, 1, 64, 3, (24, 24, 0)),
    ([3000, 700, 1500], 4, 2, 64, 16, (96, 16, 0)),     # unequal jobs: as many parts each
    ([2500], 6, 2, 32, 0, (32, 16, 0)),
    ([500], 4, 4, 256, 0, (16, 4, 0)),
    ([900, 800], 2, 1, 256, 5, (16, 8, 0)),
    ([5000, 100], 8, 2, 128, 0, (28, 7, 0)),            # parts of a single tile
    ([16384], 28, 4, 128, 0, (148, 37, 0)),             # a part an SM
    ([2000] * 74, 4, 1, 128, 0, (148, 2, 0)),
    ([3000] * 40, 1, 1, 64, 0, (280, 7, 0)),            # more parts than SMs: two teams of an SM
    ([8000] * 20, 8, 2, 128, 0, (280, 7, 0)),
    ([5000] * 10 + [5], 4, 1, 128, 0, (296, 0, 0)),     # equal shares, more ranges than SMs
    ([3000] * 4 + [20], 4, 4, 64, 16, (296, 0, 0)),
    ([600] * 20, 4, 2, 128, 0, (40, 0, 1)),             # whole jobs
]


def _range_tiles(n, first):
    """As many tokens from the first on as have the same tiles of 16."""
    return 16 * (-(-n // 16) - first // 16)


@pytest.mark.parametrize("case", CASES, ids=[f"{len(c[0])}x{max(c[0])}_q{c[1]}_kv{c[2]}_d{c[3]}" for c in CASES])
@pytest.mark.parametrize("qjl", [True, False], ids=["qjl", "plain"])
def test_ways_of_cutting(tq, oracle, case, qjl):
    lengths, q_heads, heads, dim, first, plan = case
    assert attention_plan(dim, q_heads, heads, [_range_tiles(n, first) for n in lengths]) == plan
    rng = np.random.default_rng(len(lengths) + dim)
    q = rng.standard_normal((len(lengths), q_heads, dim)).astype(np.float16)
    caches, want, want_lse = [], [], []
    for i, n in enumerate(lengths):
        k, v = kv_inputs(200 + i, n, heads, dim)
        c = tq.TQKVCache(1, heads, dim)
        c.append(0, k, v)
        caches.append(c)
        want.append(None)
        want_lse.append(None)
        if i < 2 or i == len(lengths) - 1:
            if not qjl:
                keys = np.repeat(np.asarray(c.get_keys_fp16(0, first, n), np.float64), q_heads // heads, axis=1)
                s = np.einsum("hd,thd->ht", q[i].astype(np.float64), keys) / np.sqrt(dim)
                want_lse[i] = s.max(1) + np.log(np.exp(s - s.max(1, keepdims=True)).sum(1))
            k, v = k[first:].astype(np.float32), v[first:].astype(np.float32)
            kw, kn, qw, qn = oracle.kv_encode(k, oracle.kv_seed(0, 1), oracle.kv_seed(0, 3))
            vw, vn, _, _ = oracle.kv_encode(v, oracle.kv_seed(0, 2))
            want[i] = oracle.attention(q[i].astype(np.float32), heads, kw, kn, vw, vn, qw, qn, layer=0, use_qjl=qjl)
    got, lse = tq.compressed_attention(caches, 0, q, start=first, use_qjl=qjl, return_lse=True)
    again = tq.compressed_attention(caches, 0, q, start=first, use_qjl=qjl)
    assert np.array_equal(np.asarray(got).view(np.uint16), np.asarray(again).view(np.uint16))
    for i, w in enumerate(want):
        # alone, a sequence is cut up otherwise
        alone, alone_lse = tq.compressed_attention([caches[i]], 0, q[i:i + 1], start=first, use_qjl=qjl, return_lse=True)
        assert rel_l2(got[i], alone[0].astype(np.float32)) < TOL, i
        assert np.abs(lse[i] - alone_lse[0]).max() < LSE_TOL, i
        if w is not None:
            assert rel_l2(got[i], w) < TOL, i
        if want_lse[i] is not None:
            assert np.abs(lse[i] - want_lse[i]).max() < LSE_TOL, i
    for c in caches:
        c.close()
