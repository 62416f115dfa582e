"""Writes to a decode window of more than 2^31 elements, eight at a time and one at a time: the first token, the ones around 2^31 elements, the last, and a slide past the end."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aligned", [True, False])
def test_more_elements_than_2_31(tq, aligned):
    import torch
    heads, dim, window = 8, 256, (1 << 20) + 5
    row = heads * dim
    g = torch.Generator(device="cuda").manual_seed(3)
    room = torch.zeros(window * row + 8, dtype=torch.float16, device="cuda")
    src = room[(0 if aligned else 1):][: window * row].view(window, heads, dim)
    at = [0, 1, (1 << 19) - 1, 1 << 19, (1 << 20) - 1, 1 << 20, window - 1]
    src[at] = torch.randn((len(at), heads, dim), generator=g, device="cuda").half()
    buf = tq.DecodeBuffer(window, heads, dim)
    buf.rebuild(src, src)

    def check(slot, want):
        for read in (buf.keys, buf.values):
            assert torch.equal(torch.from_numpy(read(slot, slot + 1)).view(heads, dim), want.cpu())

    for slot in at:
        check(slot, src[slot])
    check(12345, torch.zeros((heads, dim), dtype=torch.float16))
    last = src[-1].clone()
    buf.slide_window(src[: window - 1], src[: window - 1])      # (the position is now the last slot)
    ends = torch.randn((3, heads, dim), generator=g, device="cuda").half()
    buf.slide_window(ends, ends)
    for slot, want in ((window - 1, ends[0]), (0, ends[1]), (1, ends[2]), (1 << 20, src[1 << 20])):
        check(slot, want)
    assert not torch.equal(ends[0], last)
    buf.close()
