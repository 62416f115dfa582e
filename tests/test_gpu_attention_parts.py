"""Decode attention where every job (sequence, KV head, 8 query heads) is cut into as many parts as the others: a part of a single tile, parts of
unequal tiles, lengths that end inside a tile, ranges that begin inside one, jobs of other lengths beside each other, one part an SM and
two.  Against the oracle; tolerance as for the other splits of the work (test_gpu_attention_ranges)."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.golden.make_golden import kv_inputs

pytestmark = pytest.mark.gpu

TOL = 2.1e-3
CASES = [
    # tokens of each sequence, query heads, KV heads, head size, first token
    ([1024], 28, 4, 128, 0),
    ([1000, 1017], 8, 2, 128, 0),
    ([2100], 10, 1, 128, 37),              # two groups of query heads
    ([4099], 8, 1, 64, 3),
    ([3000, 700, 1500], 4, 2, 64, 16),     # unequal jobs: as many parts each
    ([2500], 6, 2, 32, 0),
    ([500], 4, 4, 256, 0),
    ([900, 800], 2, 1, 256, 5),
    ([600] * 20, 4, 2, 128, 0),            # more parts than SMs
]


@pytest.mark.parametrize("case", CASES, ids=[f"{len(c[0])}x{max(c[0])}_q{c[1]}_kv{c[2]}_d{c[3]}" for c in CASES])
@pytest.mark.parametrize("qjl", [True, False], ids=["qjl", "plain"])
def test_equal_parts(tq, oracle, case, qjl):
    lengths, q_heads, heads, dim, first = case
    rng = np.random.default_rng(len(lengths) + dim)
    q = rng.standard_normal((len(lengths), q_heads, dim)).astype(np.float16)
    caches, want = [], []
    for i, n in enumerate(lengths):
        k, v = kv_inputs(200 + i, n, heads, dim)
        c = tq.TQKVCache(1, heads, dim)
        c.append(0, k, v)
        caches.append(c)
        if i < 4 or i == len(lengths) - 1:
            k, v = k[first:].astype(np.float32), v[first:].astype(np.float32)
            kw, kn, qw, qn = oracle.kv_encode(k, oracle.kv_seed(0, 1), oracle.kv_seed(0, 3))
            vw, vn, _, _ = oracle.kv_encode(v, oracle.kv_seed(0, 2))
            want.append(oracle.attention(q[i].astype(np.float32), heads, kw, kn, vw, vn, qw, qn, layer=0, use_qjl=qjl))
        else:
            want.append(None)
    got, lse = tq.compressed_attention(caches, 0, q, start=first, use_qjl=qjl, return_lse=True)
    again = tq.compressed_attention(caches, 0, q, start=first, use_qjl=qjl)
    assert np.all(np.isfinite(lse))
    for i, w in enumerate(want):
        if w is not None:
            assert rel_l2(got[i], w) < TOL, i
    assert np.array_equal(np.asarray(got).view(np.uint16), np.asarray(again).view(np.uint16))
    for c in caches:
        c.close()
