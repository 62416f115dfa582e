"""The sums over the splits of K, at widths where the last CTA, warp or thread is not full, with fewer and with more splits than are
requested at once."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [9, 19, 75, 150])
@pytest.mark.parametrize("out", [1, 31, 128, 130, 500, 516, 1028])
def test_products_of_few_outputs(tq, rows, out):
    torch = pytest.importorskip("torch")
    cols = 4096                                            # few output tiles: K is split
    g = torch.Generator(device="cuda").manual_seed(rows + out)
    c = tq.generate_codebook(4)
    w = torch.randn((out, cols), generator=g, device="cuda") * 0.02
    lin = tq.TurboQuantLinear(cols, out, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, 128, True)), c, c, 128)
    what = torch.empty((out, cols), device="cuda")
    lin.dequantize(out=what)
    x = torch.randn((rows, cols), generator=g, device="cuda").half()
    room = torch.full((rows + 2, out), 3.0, device="cuda", dtype=torch.float16)
    y = room[1:-1]
    lin.forward(x, out=y)
    assert bool((room[0] == 3).all()) and bool((room[-1] == 3).all())
    want = x.double() @ what.double().T
    # three roundings to halves (activation, centroids, result), each of a relative size of 2^-11 / sqrt(3) at most
    assert float((y.double() - want).norm() / want.norm()) < 1e-3
    again = torch.empty_like(y)
    lin.forward(x, out=again)
    assert torch.equal(y, again)
    lin.close()
