"""Decode kernels whose columns are in several slots, two rotations: ranges of units that begin inside a slot and go on into the next.  And an infinity or a NaN in one
activation row, which shares products with the others: their bits do not change.  Tolerance: ten mantissa bits of the rotated activation and of the table, and the
result's rounding to fp16, as for three independent roundings of 2^-11 each, 2^-11 * sqrt(3 / 3), and the dequantised weights' own 2^-11."""
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _layer(tq, g, cols, rows, block, shared):
    import torch
    c = tq.generate_codebook(4)
    w = torch.randn((rows, cols), generator=g, device="cuda") * cols ** -0.5
    return tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block)


# five slots of four row tiles a unit, three, two and eight of one; row units fewer than CTAs, many more, a last one that is not whole
@pytest.mark.parametrize("cols,rows,block", [(5120, 4000, 512), (5120, 20011, 128), (11264, 2400, 512), (4608, 9000, 512), (28672, 1000, 512), (28672, 16, 1024)])
@pytest.mark.parametrize("m", [5, 8])
def test_ranges_that_cross_slots(tq, cols, rows, block, m):
    import torch
    g = torch.Generator(device="cuda").manual_seed(cols + rows + m)
    lin, other = (_layer(tq, g, cols, rows, block, False) for _ in range(2))
    x = torch.randn((m, cols), generator=g, device="cuda").half()
    back = lin.dequantize(out=torch.empty((rows, cols), device="cuda", dtype=torch.float16))
    y = lin.forward(x)
    assert rel_l2(y.cpu().numpy(), (x.double() @ back.double().T).cpu().numpy()) < 4.9e-4 + 2.0 ** -11
    assert torch.equal(tq.forward_group([lin, other], x)[0], y)
    assert torch.equal(lin.forward(x), y)
    for layer in (lin, other):
        layer.check_status()
        layer.close()


@pytest.mark.parametrize("m", [2, 3, 4, 7, 8])
@pytest.mark.parametrize("cols,block", [(1024, 128), (1536, 512), (5120, 512)])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_rows_beside_one_that_is_not_finite(tq, m, cols, block, shared, bad):
    import torch
    g = torch.Generator(device="cuda").manual_seed(cols + m)
    lin = _layer(tq, g, cols, 700, block, shared)
    x = torch.randn((m, cols), generator=g, device="cuda").half()
    clean = lin.forward(x)
    for row in range(m):
        poisoned = x.clone()
        poisoned[row, (37 * row + 5) % cols] = bad
        y = lin.forward(poisoned)
        rest = [r for r in range(m) if r != row]
        assert torch.equal(y[rest], clean[rest]) and not torch.isfinite(y[row]).any()
    lin.check_status()
    lin.close()
