"""More tokens slid into the decode window than it holds: the last ones stay, each in the slot that the tokens in order would have left it in, keys and values of one
token.  Aligned and unaligned, fp16 and fp32, device and host memory."""
import numpy as np
import pytest

from oracle.decode_window import DecodeWindow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window,heads,dim", [(1, 1, 32), (37, 3, 64), (640, 4, 128)])
@pytest.mark.parametrize("half", [True, False])
@pytest.mark.parametrize("place", ["device", "unaligned", "host", "values on the host"])
def test_slides_longer_than_the_window(tq, window, heads, dim, half, place):
    import torch
    rng = np.random.default_rng(window)
    dev, ref = tq.DecodeBuffer(window, heads, dim), DecodeWindow(window, heads, dim)

    def put(a, host):
        if host:
            return a
        room = torch.zeros(a.size + 8, dtype=torch.float16 if half else torch.float32, device="cuda")
        at = room[1:][: a.size] if place == "unaligned" else room[: a.size]
        return at.copy_(torch.from_numpy(a).cuda().flatten()).view(a.shape)

    for step, n in enumerate([window, 2, window + 1, window, 3 * window + 5, 40 * window + 3]):   # (the second moves the position)
        k, v = (rng.standard_normal((n, heads, dim)).astype(np.float16 if half else np.float32) for _ in range(2))
        move = dev.rebuild if step == 0 else dev.slide_window
        move(put(k, place == "host"), put(v, place in ("host", "values on the host")))
        (ref.rebuild if step == 0 else ref.slide_window)(k, v)
        for got, want in ((dev.keys(0, window), ref.keys(0, window)), (dev.values(0, window), ref.values(0, window))):
            assert np.array_equal(np.asarray(got).view(np.uint16).reshape(want.shape), want.view(np.uint16))
    dev.close()
