"""Linears queued one after the other behind other work, their results' places full of NaN: the bits of the same calls with a wait behind each.  Decode kernels,
products of one, two and three groups of producers, split sums."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 8, 16, 64, 128, 129, 192, 257])
@pytest.mark.parametrize("block,shared", [(128, True), (512, True), (512, False)])
def test_queued_linears(tq, m, block, shared):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    c = tq.generate_codebook(4)

    def layer(cols, rows):
        w = torch.randn((rows, cols), generator=g, device="cuda") * cols ** -0.5
        return tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block)

    several, back = [layer(3584, n) for n in (3584, 512, 512)], layer(3584, 3584)
    x = torch.randn((m, 3584), generator=g, device="cuda").half()
    stream, busy = torch.cuda.Stream(), torch.randn((4096, 4096), generator=g, device="cuda")

    def places():
        return [[torch.full((m, n), float("nan"), device="cuda", dtype=torch.float16) for n in (3584, 512, 512, 3584)] for _ in range(4)]

    def run(outs, wait):
        y = x
        for *ys, z in outs:
            tq.forward_group(several, y, outs=ys, stream=stream)
            wait()
            y = back.forward(ys[0], out=z, stream=stream)
            wait()
        return [t for row in outs for t in row]

    first = places()
    torch.cuda.synchronize()
    want = run(first, torch.cuda.synchronize)
    assert all(torch.isfinite(t).all() for t in want)
    for _ in range(3):
        outs = places()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for _ in range(8):
                busy @ busy
        got = run(outs, lambda: None)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    for lin in (*several, back):
        lin.check_status()
        lin.close()
