"""Weights with two rotations at decode sizes: one pass over pairs of fp16, scaled by powers of two."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# rounding of x, table and result to ten mantissa bits, as for one rotation
TOL = 1e-3


def layer(tq, torch, n_in, n_out, block, scale=0.02):
    g = torch.Generator(device="cuda").manual_seed(n_in + n_out + block)
    w = (torch.randn((n_out, n_in), generator=g, device="cuda") * scale).float()
    books = tq.fit_layer_codebooks(w, block, 4, 4, 20)
    qw = tq.quantize_weight(w, books[0], books[1], tq.QuantizerConfig(4, 4, block, False))
    lin = tq.TurboQuantLinear(n_in, n_out, qw, books[0], books[1], block)
    back = torch.empty((n_out, n_in), device="cuda")
    lin.dequantize(out=back)
    return lin, back.double()


# one chunk of columns and several, slices that are not full, every block size, rows that are not a whole tile
SHAPES = [(64, 40, 32), (320, 17, 64), (1024, 512, 1024), (3584, 130, 512), (4096, 48, 128), (4352, 33, 256), (9216, 100, 512), (18944, 16, 256)]


@pytest.mark.parametrize("n_in,n_out,block", SHAPES)
@pytest.mark.parametrize("rows", [1, 2, 3, 8])
def test_two_rotations_match_float64(tq, n_in, n_out, block, rows):
    torch = pytest.importorskip("torch")
    lin, w = layer(tq, torch, n_in, n_out, block)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, n_in), generator=g, device="cuda").half()
    want = x.double() @ w.T
    y = lin.forward(x)
    assert rel_l2(y.double().cpu(), want.cpu()) < TOL
    # an activation that is not 16-byte aligned: the same bits
    shifted = torch.empty(rows * n_in + 1, device="cuda", dtype=torch.float16)[1:].view(rows, n_in).copy_(x)
    assert torch.equal(lin.forward(shifted), y)
    # a group of layers: the same bits as the layers alone
    other, _ = layer(tq, torch, n_in, n_out + 16, block)
    group = tq.forward_group([other, lin], x)
    assert torch.equal(group[0], other.forward(x)) and torch.equal(group[1], y)
    lin.check_status()


@pytest.mark.parametrize("exponent", [-9, 12])
def test_two_rotations_at_other_magnitudes(tq, exponent):
    """The scales are powers of two: they cannot be seen in a result that is not itself rounded differently.  Rows and slices
    of different magnitude do not disturb one another."""
    torch = pytest.importorskip("torch")
    lin, w = layer(tq, torch, 1024, 96, 128)
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn((4, 1024), generator=g, device="cuda").half()
    x = torch.where(x.abs() < 2.0 ** -4, torch.ones_like(x), x)   # (no subnormal numbers after scaling)
    y = lin.forward(x)
    xs = x.clone()
    xs[1] *= 2.0 ** exponent
    ys = lin.forward(xs)
    for r in (0, 2, 3):
        assert torch.equal(ys[r], y[r])
    assert rel_l2(ys[1].double().cpu(), (xs[1].double() @ w.T).cpu()) < TOL
    scaled = y[1].float() * 2.0 ** exponent
    normal = (y[1].abs() >= 2.0 ** -14) & (scaled.abs() >= 2.0 ** -14)
    assert int(normal.sum()) > 80 and torch.equal(ys[1].float()[normal], scaled[normal])
    mixed = x.clone()
    mixed[:, 256:512] *= 2.0 ** exponent   # one slice of 256 columns
    want = mixed.double() @ w.T
    assert rel_l2(lin.forward(mixed).double().cpu(), want.cpu()) < TOL


def test_two_rotations_zero_and_infinite_rows(tq):
    torch = pytest.importorskip("torch")
    lin, w = layer(tq, torch, 512, 64, 128)
    x = torch.zeros((3, 512), device="cuda", dtype=torch.float16)
    x[1] = 1.0
    x[2, 7] = float("inf")
    y = lin.forward(x)
    assert torch.equal(y[0], torch.zeros_like(y[0]))
    assert rel_l2(y[1].double().cpu(), (x[1].double() @ w.T).cpu()) < TOL
    assert not torch.isfinite(y[2]).any()


@pytest.mark.parametrize("rows", [1, 5, 40])
@pytest.mark.parametrize("odd", [float("inf"), float("nan")])
def test_two_rotations_beside_a_centroid_that_is_not_finite(tq, rows, odd):
    """A codebook entry that no weight uses, or one row alone, does not change the other rows, however small their centroids are."""
    torch = pytest.importorskip("torch")
    n_in, n_out, block = 512, 48, 128
    rng = np.random.default_rng(rows)
    primary = (np.sort(rng.standard_normal(16)) * 1e-6).astype(np.float32)
    residual = (np.sort(rng.standard_normal(16)) * 1e-7).astype(np.float32)
    primary[15] = odd
    code = rng.integers(0, 15, (n_out, n_in))
    code[7] = 15
    other = rng.integers(0, 16, (n_out, n_in))
    pack = lambda c: (c[:, 0::2] | (c[:, 1::2] << 4)).astype(np.uint8)
    qw = tq.QuantizedWeight(pack(code), pack(other), np.full(n_out, 1e6, np.float32), np.array([11, 12, block], np.uint32))
    lin = tq.TurboQuantLinear(n_in, n_out, qw, tq.codebook_from_centroids(primary), tq.codebook_from_centroids(residual), block)
    back = torch.empty((n_out, n_in), device="cuda")
    lin.dequantize(out=back)
    x = torch.randn((rows, n_in), generator=torch.Generator(device="cuda").manual_seed(rows), device="cuda").half()
    y = lin.forward(x)
    keep = torch.arange(n_out, device="cuda") != 7
    want = x.double() @ back[keep].double().T
    assert rel_l2(y[:, keep].double().cpu(), want.cpu()) < TOL
    assert not torch.isfinite(y[:, 7]).any()
    lin.close()
