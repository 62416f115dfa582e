"""Window attention on either side of the size from which the window is read past the first-level cache (60 MB), token counts that end inside a tile.
Tolerance: scores of fp16 operands are summed in fp32 and exponentials rounded to fp16, 2^-11 each; the result is rounded to fp16: as for three independent
roundings, 2^-11 * sqrt(3 / 3)."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [30720, 30721, 30739])    # 30720 tokens of 4 heads of 128: 60 MB
@pytest.mark.parametrize("half", [True, False])
def test_window_around_the_streamed_size(tq, tokens, half):
    import torch
    g = torch.Generator(device="cuda").manual_seed(tokens)
    k, v = (torch.randn((tokens, 4, 128), generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn((28, 128), generator=g, device="cuda").half()
    window, cache = tq.DecodeBuffer(tokens, 4, 128), tq.TQKVCache(1, 4, 128)
    cache.append(0, k, v)
    window.rebuild(k, v)
    got = tq.hybrid_attention(cache, window, 0, q if half else q.float())
    want = np.empty((28, 128))
    for h in range(28):
        p = torch.softmax(k[:, h // 7].double() @ q[h].double() / 128 ** 0.5, 0)
        want[h] = (p @ v[:, h // 7].double()).cpu().numpy()
    assert rel_l2(got.cpu().numpy().reshape(28, 128), want) < 4.9e-4
    cache.close()
