"""Decode attention against the oracle at the batches where the split of its work changes: jobs cut over many thread-block
teams (one long sequence, few heads), whole jobs per team (one and several each), unequal lengths, more sequences than travel
as kernel parameters.  Tolerance: the query is rounded to fp16, 2^-12 of a value in the root mean square, which moves a
score s by up to 2^-12 |s| and its probability by as much relatively; with the inputs' outlier channels the scores that count
reach about 8, so 2.0e-3; the result's rounding adds 2.4e-4 in squares."""
import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.golden.make_golden import kv_inputs

pytestmark = pytest.mark.gpu

TOL = 2.1e-3
CASES = [
    # tokens of each sequence, query heads, KV heads, head size
    ([6000], 4, 1, 32),                       # many parts of one job
    ([9000], 8, 1, 128),
    ([5000, 17], 2, 1, 64),
    ([1500], 3, 1, 256),
    ([40] * 9, 8, 2, 128),                    # whole jobs, one per team
    ([33, 1, 16, 90, 15, 47] * 6, 18, 2, 64),     # ... a group of 8 heads and one of a single head, lengths mixed
    ([20, 5, 64] * 34, 4, 4, 128),            # ... two per team, descriptors from a table
]


@pytest.mark.parametrize("case", CASES, ids=[f"{len(c[0])}x{max(c[0])}_q{c[1]}_kv{c[2]}_d{c[3]}" for c in CASES])
@pytest.mark.parametrize("qjl", [True, False], ids=["qjl", "plain"])
def test_attention_work_split(tq, oracle, case, qjl):
    lengths, q_heads, heads, dim = case
    rng = np.random.default_rng(len(lengths) + dim)
    q = rng.standard_normal((len(lengths), q_heads, dim)).astype(np.float16)
    caches, want = [], []
    for i, n in enumerate(lengths):
        k, v = kv_inputs(100 + i, n, heads, dim)
        c = tq.TQKVCache(1, heads, dim)
        c.append(0, k, v)
        caches.append(c)
        if i < 8 or i >= len(lengths) - 4:    # the oracle's share of a large batch: its ends
            kw, kn, qw, qn = oracle.kv_encode(k.astype(np.float32), oracle.kv_seed(0, 1), oracle.kv_seed(0, 3))
            vw, vn, _, _ = oracle.kv_encode(v.astype(np.float32), oracle.kv_seed(0, 2))
            want.append(oracle.attention(q[i].astype(np.float32), heads, kw, kn, vw, vn, qw, qn, layer=0, use_qjl=qjl))
        else:
            want.append(None)
    got = tq.compressed_attention(caches, 0, q, use_qjl=qjl)
    again = tq.compressed_attention(caches, 0, q, use_qjl=qjl)
    for i, w in enumerate(want):
        if w is not None:
            assert rel_l2(got[i], w) < TOL, i
        assert rel_l2(got[i], tq.compressed_attention([caches[i]], 0, q[i:i + 1], use_qjl=qjl)[0].astype(np.float32)) < TOL, i
    assert np.array_equal(np.asarray(got).view(np.uint16), np.asarray(again).view(np.uint16))
    for c in caches:
        c.close()


def encoded(tq, oracle, k, v):
    heads, dim = k.shape[1:]
    c = tq.TQKVCache(1, heads, dim)
    c.append(0, k, v)
    kw, kn, qw, qn = oracle.kv_encode(k, oracle.kv_seed(0, 1), oracle.kv_seed(0, 3))
    vw, vn, _, _ = oracle.kv_encode(v, oracle.kv_seed(0, 2))
    return c, (kw, kn, vw, vn, qw, qn)


@pytest.mark.parametrize("dim", [32, 64, 128, 256])
@pytest.mark.parametrize("norm", [1e-6, 1e-3, 1e4, 5e4])
def test_attention_takes_any_value_norm(tq, oracle, dim, norm):
    """Value norms at both ends of what an fp16 result can hold, some of them zero: the largest weight times norm is brought
    into fp16's range whatever it is."""
    heads, q_heads, n = 2, 6, 700
    k, v = (t.astype(np.float32) for t in kv_inputs(dim, n, heads, dim))
    v *= norm / np.linalg.norm(v, axis=-1).mean()
    v[5:9] = 0.0
    v[40:60] *= 1e-3
    c, codes = encoded(tq, oracle, k, v)
    q = np.random.default_rng(dim).standard_normal((1, q_heads, dim)).astype(np.float16)
    got, lse = tq.compressed_attention([c], 0, q, use_qjl=True, return_lse=True)
    want = oracle.attention(q[0].astype(np.float32), heads, *codes, layer=0, use_qjl=True)
    assert np.all(np.isfinite(got.astype(np.float32))) and np.all(np.isfinite(lse))
    off = np.linalg.norm(got[0].astype(np.float64) - want)
    assert off < TOL * np.linalg.norm(want) + 2.0 ** -25 * np.sqrt(want.size), off   # half of fp16's smallest step
    c.close()


@pytest.mark.parametrize("dim", [32, 64, 128, 256])
@pytest.mark.parametrize("scale", [1e-4, 1e4])
def test_attention_takes_any_query_scale(tq, oracle, dim, scale):
    """Queries near the ends of fp16's range against keys of the inverse scale: the rotated query, and the query with the
    residual's signs, keep all their bits."""
    heads, q_heads, n = 2, 6, 700
    k, v = (t.astype(np.float32) for t in kv_inputs(dim, n, heads, dim))
    c, codes = encoded(tq, oracle, (k / np.float32(scale)), v)
    q = (np.random.default_rng(dim).standard_normal((1, q_heads, dim)) * scale).astype(np.float16)
    got = tq.compressed_attention([c], 0, q, use_qjl=True)
    want = oracle.attention(q[0].astype(np.float32), heads, *codes, layer=0, use_qjl=True)
    # without the scaling 8e-4 at 128 dims and 4e-4 to 1.1e-3 at the others, with it what a scale of one has
    assert rel_l2(got[0], want) < (7e-4 if dim == 128 else 4e-4)
    c.close()


@pytest.mark.parametrize("dim", [32, 64, 256])
@pytest.mark.parametrize("n", [40, 5000])
def test_other_head_sizes_are_multiplied_as_fp32(tq, oracle, dim, n):
    """The softmax denominator of head sizes other than 128 against double sums over the stored codes.  Scores reach 30: an
    fp32 sum of them is good to 2^-24 x 30 per step, a few steps; centroids in plain fp16 left 1e-4."""
    heads, q_heads = 2, 6
    k, v = (t.astype(np.float32) for t in kv_inputs(n + dim, n, heads, dim))
    q = np.random.default_rng(dim).standard_normal((1, q_heads, dim)).astype(np.float16)
    k[n // 3] = 2.0 * q[0, ::q_heads // heads].astype(np.float32)          # one key that stands out
    c, (kw, kn, vw, vn, qw, qn) = encoded(tq, oracle, k, v)
    out, lse = tq.compressed_attention([c], 0, q, use_qjl=True, return_lse=True)
    cents = oracle.codebook(3)[0].astype(np.float64)
    d = np.arange(dim)
    codes = (kw[:, d // 10] >> (3 * (d % 10)).astype(np.uint32)) & 7
    signs = ((qw[:, d // 32] >> (d % 32).astype(np.uint32)) & 1) * 2.0 - 1.0
    rot = oracle.wht(q[0].astype(np.float32), oracle.kv_seed(0, 1), dim).astype(np.float64)
    flip = np.array([1.0 if (oracle.kv_seed(0, 3) * 2654435761 + j * 2246822519) >> 31 & 1 else -1.0 for j in range(dim)])
    for h in range(q_heads):
        own = slice(h // (q_heads // heads), None, heads)                  # records of the KV head
        r = rot[h]
        dot = cents[codes[own]] @ r + np.sqrt(2 / (np.pi * dim)) * qn[own].astype(np.float64) * (signs[own] @ (flip * r))
        s = dot * kn[own].astype(np.float64) / dim
        want = s.max() + np.log(np.exp(s - s.max()).sum())
        assert abs(lse[0, h] - want) < 1e-5, (h, lse[0, h], want)
    want = oracle.attention(q[0].astype(np.float32), heads, kw, kn, vw, vn, qw, qn, layer=0, use_qjl=True)
    assert rel_l2(out[0], want) < 4e-4                                     # the result's rounding: 2^-12 in the mean
    c.close()
