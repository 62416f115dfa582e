"""Window attention on either side of the size from which the window is read past the first-level cache (five sixths of the L2 cache), token counts that end inside a
tile, one window again and two in turn.  Tolerance: scores of fp16 operands are summed in fp32 and exponentials rounded to fp16, 2^-11 each; the result is rounded to
fp16: as for three independent roundings, 2^-11 * sqrt(3 / 3)."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beyond", [-37, 0, 1, 37])   # tokens more than five sixths of the cache hold
@pytest.mark.parametrize("heads", [1, 4])
@pytest.mark.parametrize("half", [True, False])
def test_window_around_the_cache_size(tq, beyond, heads, half):
    import torch
    tokens = torch.cuda.get_device_properties(0).L2_cache_size // 6 * 5 // (heads * 128 * 4) + beyond
    g = torch.Generator(device="cuda").manual_seed(tokens)
    q = torch.randn((7 * heads, 128), generator=g, device="cuda").half()
    sides = []
    for _ in range(2):
        k, v = (torch.randn((tokens, heads, 128), generator=g, device="cuda").half() for _ in range(2))
        window, cache = tq.DecodeBuffer(tokens, heads, 128), tq.TQKVCache(1, heads, 128)
        cache.append(0, k, v)
        window.rebuild(k, v)
        want = np.empty((7 * heads, 128))
        for h in range(7 * heads):
            p = torch.softmax(k[:, h // 7].double() @ q[h].double() / 128 ** 0.5, 0)
            want[h] = (p @ v[:, h // 7].double()).cpu().numpy()
        sides.append((cache, window, want))
    for i in (0, 0, 1, 0, 1):
        cache, window, want = sides[i]
        got = tq.hybrid_attention(cache, window, 0, q if half else q.float())
        assert rel_l2(got.cpu().numpy().reshape(want.shape), want) < 4.9e-4
    for cache, window, _ in sides:
        cache.close()
        window.close()
