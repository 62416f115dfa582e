"""The encoder of long appends against the one of a decode step's few vectors (which has its own way through codes, signs and
sums): the stored bits are the same, for odd starts and lengths, and for vectors that are not ordinary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("dtype", ["f16", "f32"])
@pytest.mark.parametrize("first,tokens,heads,shift", [(0, 1300, 1, 0), (1, 1299, 1, 0), (3, 650, 2, 1), (0, 320, 5, 0)])
def test_long_appends_store_what_short_ones_do(tq, dim, dtype, first, tokens, heads, shift):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(tokens + dim)
    kind = torch.float16 if dtype == "f16" else torch.float32

    def vectors(n):
        room = torch.zeros(n * heads * dim + shift, device="cuda", dtype=kind)   # (shift: not on a 16-byte boundary)
        x = torch.randn((n, heads, dim), generator=g, device="cuda")
        x[1::7] *= 1e-3
        x[2::7] = 0.0
        x[3::11, :, ::2] = 0.0
        x[4::13] = 1.0
        if n > 40:
            x[30, 0, 5] = float("inf")
            x[31, 0, 6] = float("nan")
        return room[shift:].view(n, heads, dim).copy_(x)

    lead_k, lead_v, k, v = vectors(max(first, 1)), vectors(max(first, 1)), vectors(tokens), vectors(tokens)
    long, short = tq.TQKVCache(1, heads, dim), tq.TQKVCache(1, heads, dim)
    for cache in (long, short):
        if first:
            cache.append(0, lead_k, lead_v)
    long.append(0, k, v)
    step = 37
    for t in range(0, tokens, step):
        short.append(0, k[t:t + step], v[t:t + step])
    a, b = long.export(0), short.export(0)
    for name in a:
        if name != "tokens":
            assert np.array_equal(a[name], b[name], equal_nan=a[name].dtype == np.float32), name


@pytest.mark.parametrize("dim", [32, 64, 128, 256, 512])
@pytest.mark.parametrize("heads", [1, 3])
def test_decoded_ranges_of_any_length_and_place(tq, dim, heads):
    """Results that do not fill a warp's eight vectors, and ones that are not on a 16-byte boundary: the same bits."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(dim)
    k = torch.randn((101, heads, dim), generator=g, device="cuda").half()
    v = torch.randn((101, heads, dim), generator=g, device="cuda").half()
    cache = tq.TQKVCache(1, heads, dim)
    cache.append(0, k, v)
    for get, src in ((cache.get_keys_fp16, k), (cache.get_values_fp16, v)):
        whole = torch.empty((101, heads, dim), device="cuda", dtype=torch.float16)
        get(0, 0, 101, out=whole)
        assert float((whole.double() - src.double()).norm() / src.double().norm()) < 0.25   # three bits
        for start, end in ((0, 1), (5, 6), (3, 12), (16, 33), (100, 101), (1, 100)):
            n = (end - start) * heads * dim
            room = torch.full((n + 16,), 3.0, device="cuda", dtype=torch.float16)
            for at in (0, 1, 8):
                room.fill_(3.0)
                out = room[at:at + n].view(end - start, heads, dim)
                get(0, start, end, out=out)
                assert torch.equal(out, whole[start:end])
                assert bool((room[:at] == 3).all()) and bool((room[at + n:] == 3).all())
