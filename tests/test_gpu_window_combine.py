"""The sum of the window attention's splits: every head size, from one split to the most there are, counts that fill the rows of
a block and counts that do not."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,group,dim,tokens", [
    (1, 1, 128, 100),        # one split
    (1, 3, 64, 128 * 5 + 1),
    (2, 7, 128, 128 * 33),
    (4, 7, 128, 14208),      # 111 splits
    (1, 8, 32, 128 * 255),
    (1, 2, 256, 128 * 256 + 77),   # as many splits as there may be
    (1, 1, 128, 40000),
])
def test_window_attention_over_many_splits(tq, heads, group, dim, tokens):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(tokens)
    k = torch.randn((tokens, heads, dim), generator=g, device="cuda").half()
    v = torch.randn((tokens, heads, dim), generator=g, device="cuda").half()
    q = (4 * torch.randn((heads * group, dim), generator=g, device="cuda")).half()   # a few tokens carry most of the weight
    cache, window = tq.TQKVCache(1, heads, dim), tq.DecodeBuffer(tokens, heads, dim)
    cache.append(0, k, v)
    window.rebuild(k, v)
    out = tq.hybrid_attention(cache, window, 0, q)
    torch.cuda.synchronize()
    s = torch.einsum("hgd,thd->hgt", q.double().view(heads, group, dim), k.double()) / dim ** 0.5
    want = torch.einsum("hgt,thd->hgd", torch.softmax(s, -1), v.double()).reshape(heads * group, dim)
    # weights and results are rounded to fp16: 2^-12 of a value each on average, not more than twice that together
    assert rel_l2(out.float().cpu().numpy() if hasattr(out, "cpu") else np.asarray(out), want.cpu().numpy()) < 2 * 2.0 ** -11
