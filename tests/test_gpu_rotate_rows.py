"""The activation rotation of the many-row linear at the edges of its tiles: blocks of 32 to 1024 columns, a last group of columns
that is not full, rows around the groups of 8 and 32, several steps per CTA.
Tolerance as in test_gpu_gemm_edges: three roundings to fp16, root mean square below 4.9e-4; a row on its own may reach 1.5 of that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,block,shared", [
    (64, 32, True), (192, 64, False), (320, 64, True), (3584, 128, True), (384, 128, False), (768, 256, True), (1536, 512, False),
    (512, 512, True), (2048, 1024, False),
])
@pytest.mark.parametrize("rows", [9, 31, 33, 257])
def test_rotation_of_many_rows(tq, n_in, block, shared, rows):
    check(tq, n_in, block, shared, rows)


@pytest.mark.parametrize("n_in,block,rows", [(8192, 64, 1300), (16384, 128, 2050), (16384, 512, 2077)])
def test_rotation_with_several_steps(tq, n_in, block, rows):
    check(tq, n_in, block, True, rows)


@pytest.mark.parametrize("n_in,block,shared", [
    (64, 32, True), (192, 64, False), (128, 128, True), (3584, 128, True), (768, 256, False), (512, 512, True), (1536, 512, False), (1024, 1024, True),
])
def test_alignment_does_not_show(tq, n_in, block, shared):
    """An activation that is not 16-byte aligned is rotated by another kernel, which adds in the same order: the same bits, also
    where the sums of a block have to be rounded (values of very different size)."""
    torch = pytest.importorskip("torch")
    rows, n_out = 300, 256
    g = torch.Generator(device="cuda").manual_seed(n_in + block)
    c = tq.generate_codebook(4)
    w = torch.randn((n_out, n_in), generator=g, device="cuda") * 0.02
    lin = tq.TurboQuantLinear(n_in, n_out, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block)
    x = torch.randn((rows, n_in), generator=g, device="cuda")
    x = (x * 2.0 ** torch.randint(-16, 6, x.shape, generator=g, device="cuda")).half()
    shifted = torch.empty(rows * n_in + 1, device="cuda", dtype=torch.float16)[1:].view(rows, n_in).copy_(x)
    y = lin.forward(x)
    assert torch.isfinite(y).all()
    assert torch.equal(lin.forward(shifted), y)
    lin.check_status()
    lin.close()


def check(tq, n_in, block, shared, rows):
    torch = pytest.importorskip("torch")
    n_out = 144
    g = torch.Generator(device="cuda").manual_seed(n_in + block + rows)
    w = torch.randn((n_out, n_in), generator=g, device="cuda") * 0.02
    c = tq.generate_codebook(4)
    layers = []
    for _ in range(2):
        qw = tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared))
        layers.append(tq.TurboQuantLinear(n_in, n_out, qw, c, c, block))
        w = torch.randn((n_out, n_in), generator=g, device="cuda") * 0.02
    x = torch.randn((rows, n_in), generator=g, device="cuda").half()
    alone = [lin.forward(x) for lin in layers]
    for lin, y in zip(layers, alone):
        back = torch.empty((n_out, n_in), device="cuda")
        lin.dequantize(out=back)
        want = x.double() @ back.double().T
        err = (y.double() - want).norm(dim=1) / want.norm(dim=1)
        assert float(err.square().mean().sqrt()) < 4.9e-4
        assert float(err.max()) < 1.5 * 4.9e-4
        lin.check_status()
    for y, got in zip(alone, tq.forward_group(layers, x)):
        assert torch.equal(y, got)


@pytest.mark.parametrize("n_in,n_out,rows,stride", [
    (3584, 1024, 64, 0), (4096, 130, 40, 0), (4096, 126, 9, 0), (2048, 128, 300, 0),   # rows of four outputs, and not
    (4096, 128, 17, 131), (4096, 128, 17, 136),                                        # rows of a wider buffer
    (8192, 16, 65, 0),                                                                 # more than eight splits
])
def test_sums_over_the_splits_of_k(tq, n_in, n_out, rows, stride):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(n_in + n_out + rows)
    w = torch.randn((n_out, n_in), generator=g, device="cuda") * 0.02
    c = tq.generate_codebook(4)
    lin = tq.TurboQuantLinear(n_in, n_out, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, 128, True)), c, c, 128)
    back = torch.empty((n_out, n_in), device="cuda")
    lin.dequantize(out=back)
    x = torch.randn((rows, n_in), generator=g, device="cuda").half()
    y = lin.forward(x)
    want = x.double() @ back.double().T
    assert float((y.double() - want).norm() / want.norm()) < 4.9e-4
    if stride:
        wide = torch.full((rows, stride), 7.0, device="cuda", dtype=torch.float16)
        lin.forward_strided(x, wide.data_ptr() + 2 * 3, stride)
        torch.cuda.synchronize()
        assert torch.equal(wide[:, 3:3 + n_out], y) and bool((wide[:, :3] == 7).all()) and bool((wide[:, 3 + n_out:] == 7).all())
    lin.check_status()
