"""The decode window's writes eight elements at a time, and element by element where rows or pointers are not whole 16-byte pieces: wrapped around the
ring's end, of fp16 and fp32, the same values."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim", [(1, 32), (3, 64), (4, 128), (2, 256)])
@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("shift", [0, 1])
def test_window_writes(tq, heads, dim, half, shift):
    import torch
    g = torch.Generator(device="cuda").manual_seed(dim)
    window, row = 37, heads * dim
    buf = tq.DecodeBuffer(window, heads, dim)

    def rows(n):
        room = torch.randn((2, n * row + 8), generator=g, device="cuda").to(torch.float16 if half else torch.float32)
        return [r[shift:][: n * row].view(n, heads, dim) for r in room]

    k, v = rows(window)
    buf.rebuild(k, v)
    kept = [k.half().clone(), v.half().clone()]
    for step in range(20):   # three slots at a time, past the ring's end
        k, v = rows(3)
        buf.slide_window(k, v)
        at = [(3 * step + t) % window for t in range(3)]
        for a, b in zip(kept, (k, v)):
            a[at] = b.half()
    for got, want in zip((buf.keys(0, window), buf.values(0, window)), kept):
        assert torch.equal(torch.as_tensor(got).cuda().half().view(window, heads, dim), want)
    k, v = rows(5)
    buf.rebuild(k, v)
    for got, want in zip((buf.keys(0, 5), buf.values(0, 5)), (k.half(), v.half())):
        assert torch.equal(torch.as_tensor(got).cuda().half().view(5, heads, dim), want)
