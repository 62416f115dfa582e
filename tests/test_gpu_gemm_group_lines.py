"""Several matrices of more than 128 rows with two groups of producers and with three: stages of the longest CTAs around the line between them, one K split and more, equal
splits and unequal ones.  Up to 128 rows: one group, two and three, waves of equal CTAs and sums of unequal ones around the lines between them.  And, of one matrix with two
rotations, the lines between two groups and three.  Tolerance: three independent roundings to fp16,
2^-11 * sqrt(3 / 3), and the dequantised weights' own 2^-11."""
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _layer(tq, g, cols, rows, shared):
    import torch
    c = tq.generate_codebook(4)
    w = torch.randn((rows, cols), generator=g, device="cuda") * cols ** -0.5
    return tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, 64, shared)), c, c, 64)


def _check(lin, x, y):
    import torch
    back = lin.dequantize(out=torch.empty((lin.out_features(), lin.in_features()), device="cuda", dtype=torch.float16))
    assert rel_l2(y.cpu().numpy(), (x.double() @ back.double().T).cpu().numpy()) < 4.9e-4 + 2.0 ** -11
    lin.check_status()


# 50 tiles of a token tile: two splits, one with two token tiles
@pytest.mark.parametrize("stages", [25, 26, 27, 28])
@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("outs", [(6400, 130, 128), (130, 6400), (6400, 6399)])
@pytest.mark.parametrize("m,shared", [(129, False), (256, False), (257, False), (200, True)])
def test_long_and_short_ctas(tq, stages, odd, outs, m, shared):
    import torch
    g = torch.Generator(device="cuda").manual_seed(stages + m)
    cols = 64 * (2 * stages * (2 if shared else 1) - odd)
    lins = [_layer(tq, g, cols, out, shared) for out in outs]
    x = torch.randn((m, cols), generator=g, device="cuda").half()
    for lin, y in zip(lins, tq.forward_group(lins, x)):
        _check(lin, x, y)
        assert torch.equal(lin.forward(x), y)
        lin.close()


# (a stage is one 64-column block here; 80 tiles: K is not split)
@pytest.mark.parametrize("m,stages", [(20, 29), (20, 30), (20, 31), (32, 30), (32, 31), (33, 23), (33, 24), (33, 25), (100, 24), (100, 25)])
def test_two_rotations_around_the_line_between_two_groups_and_three(tq, m, stages):
    import torch
    g = torch.Generator(device="cuda").manual_seed(stages + m)
    lin = _layer(tq, g, 64 * stages, 128 * 80, False)
    x = torch.randn((m, 64 * stages), generator=g, device="cuda").half()
    _check(lin, x, lin.forward(x))
    lin.close()


# 150 tiles each: three waves of CTAs alone on an SM or two of two to an SM, one group up to 20 stages; 146 and 150: one wave of two to an SM
@pytest.mark.parametrize("stages", [19, 20, 21, 22])
@pytest.mark.parametrize("outs", [(19200, 19200), (19200, 18561), (18688, 19200)])
@pytest.mark.parametrize("m,shared", [(16, True), (64, True), (65, True), (32, False), (33, False), (128, False)])
def test_waves_up_to_128_rows(tq, stages, outs, m, shared):
    import torch
    g = torch.Generator(device="cuda").manual_seed(stages + m)
    cols = 64 * stages * (2 if shared else 1)
    lins = [_layer(tq, g, cols, out, shared) for out in outs]
    x = torch.randn((m, cols), generator=g, device="cuda").half()
    for lin, y in zip(lins, tq.forward_group(lins, x)):
        _check(lin, x, y)
        lin.close()


# 64 tiles in two splits beside 8 in up to 18: one group while the long CTAs are short
@pytest.mark.parametrize("k_blocks", [60, 74, 78, 79, 80, 90])
@pytest.mark.parametrize("m", [16, 32, 64, 128])
def test_unequal_ctas_up_to_128_rows(tq, k_blocks, m):
    import torch
    g = torch.Generator(device="cuda").manual_seed(k_blocks + m)
    lins = [_layer(tq, g, 64 * k_blocks, out, False) for out in (8192, 1024, 1000)]
    x = torch.randn((m, 64 * k_blocks), generator=g, device="cuda").half()
    for lin, y in zip(lins, tq.forward_group(lins, x)):
        _check(lin, x, y)
        assert torch.equal(lin.forward(x), y)
        lin.close()
