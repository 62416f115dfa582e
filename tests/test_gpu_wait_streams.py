"""A wait for a late rank leaves the GPU to other streams: the kernels behind it do not come before it is over, so linears of another stream run to their end meanwhile,
and the wait's own stream gives the bits of the same calls without one.  The other rank is the host here: it copies the flag, or the packets, when the other stream is done."""
import time

import pytest

from tests.test_gpu_late_exchange import _Late, _layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["flags", "packets", "sums", "sums+norm"])
@pytest.mark.parametrize("m", [1, 16, 64])   # decode kernels; products of two producer groups (of one, several at once) with their tensor memory
def test_other_streams_run_beside_a_wait(tq, kind, m):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    mine, other = ([_layer(tq, g, 3584, out) for out in (3584, 512, 512)] for _ in range(2))
    x = torch.randn((m, 3584), generator=g, device="cuda").half()
    streams = [torch.cuda.Stream() for _ in range(2)]

    def calls(layers, stream):
        return [*tq.forward_group(layers, x, stream=stream), layers[0].forward(x, stream=stream)]

    want = [calls(layers, stream) for layers, stream in zip((mine, other), streams)]
    torch.cuda.synchronize()
    late = _Late(tq, kind, g)
    late.wait(streams[0])
    got = [calls(mine, streams[0]), calls(other, streams[1])]
    until = time.monotonic() + 0.4                    # (the wait's own limit is a second)
    while not streams[1].query() and time.monotonic() < until:
        pass
    done, waiting = streams[1].query(), not streams[0].query()
    late.arrive()
    torch.cuda.synchronize()
    for layer in (*mine, *other):
        layer.check_status()
        layer.close()
    late.close()
    assert done and waiting
    for a, b in zip(got, want):
        assert all(torch.equal(p, q) for p, q in zip(a, b))
