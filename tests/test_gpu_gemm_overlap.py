"""Many-row linears with one, two and three groups of producers: the lines between them, and the counts of split sums at which the kernel that adds
them changes.  (Chains of dependent calls, whose kernels are set up beside the ones in front: test_gpu_ordering.py.)  Tolerance: three
independent roundings to fp16, 2^-11 * sqrt(3 / 3), and the dequantised weights' own."""
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _layer(tq, g, cols, rows, block=128, shared=True):
    import torch
    c = tq.generate_codebook(4)
    w = torch.randn((rows, cols), generator=g, device="cuda") * cols ** -0.5
    return tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block)


def _check(lin, x):
    import torch
    back = lin.dequantize(out=torch.empty((lin.out_features(), lin.in_features()), device="cuda", dtype=torch.float16))
    y = lin.forward(x)
    assert rel_l2(y.cpu().numpy(), (x.double() @ back.double().T).cpu().numpy()) < 4.9e-4 + 2.0 ** -11
    lin.check_status()
    return y


@pytest.mark.parametrize("splits", [2, 8, 9, 12, 16, 17, 25])
@pytest.mark.parametrize("rows", [64, 127])     # whole pieces of four results, and not
@pytest.mark.parametrize("m", [10, 70])
def test_counts_of_split_sums(tq, splits, rows, m):
    import torch
    g = torch.Generator(device="cuda").manual_seed(splits + m)
    lin = _layer(tq, g, 64 * 8 * splits, rows)
    _check(lin, torch.randn((m, 64 * 8 * splits), generator=g, device="cuda").half())
    lin.close()


# K blocks of a CTA around the line between two groups of producers and three, up to 32 rows and above; 80 tiles: K is not split
@pytest.mark.parametrize("k_blocks", [47, 48, 49, 50, 59, 60, 61, 62])
@pytest.mark.parametrize("m,shared", [(32, True), (33, True), (20, False)])
def test_stages_around_the_line_between_two_groups_and_three(tq, k_blocks, m, shared):
    import torch
    g = torch.Generator(device="cuda").manual_seed(k_blocks + m)
    lin = _layer(tq, g, 64 * k_blocks, 128 * 80, 64, shared)
    _check(lin, torch.randn((m, 64 * k_blocks), generator=g, device="cuda").half())
    lin.close()


# CTAs of several matrices around the number of SMs, rows around what one group of producers takes and around the tensor memory's division for it
@pytest.mark.parametrize("m", [15, 64, 65, 128, 129])
@pytest.mark.parametrize("outs,shared", [((128 * 74, 128 * 74), True), ((128 * 74, 128 * 75), True), ((128 * 100, 128 * 197), True), ((130, 128 * 148), False)])
def test_several_matrices_of_one_group(tq, outs, m, shared):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    lins = [_layer(tq, g, 320, o, 64, shared) for o in outs]
    x = torch.randn((m, 320), generator=g, device="cuda").half()
    for lin, y in zip(lins, tq.forward_group(lins, x)):
        assert torch.equal(y, _check(lin, x))
    for lin in lins:
        lin.close()
