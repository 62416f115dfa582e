"""The many-row linear's three groups of dequantising warps: fewer stages (128 columns each, 64 with two rotations) than groups, one and two
more than a multiple of three, a last stage of one K block, and the stages of several tiles running on through the ring.  Tolerance: as at
the tile edges, three independent roundings to fp16, 2^-11 * sqrt(3 / 3)."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

# columns, weight rows, activation rows, shared rotation
CASES = [(64 * k, 130, 9 + 60 * k, k % 3 != 0) for k in range(1, 12)]
CASES += [(128, 38000, 9, True), (192, 38000, 65, True), (448, 19100, 129, True), (128, 19100, 40, False), (320, 19100, 256, True)]


@pytest.mark.parametrize("cols,rows,m,shared", CASES)
def test_stages_and_groups(tq, oracle, cols, rows, m, shared):
    import torch
    rng = np.random.default_rng(rows + cols + m)
    cb = oracle.codebook(4)[0]
    w = (rng.standard_normal((rows, cols)) * 0.02).astype(np.float16).astype(np.float32)
    pp, pr, norms, seeds = oracle.quantize_weight(w, cb, cb, 4, 4, 64, shared)
    x = rng.standard_normal((m, cols)).astype(np.float16)
    c = tq.codebook_from_centroids(cb)
    lin = tq.TurboQuantLinear(cols, rows, tq.QuantizedWeight(pp, pr, norms, seeds), c, c, 64)
    y = lin.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    assert rel_l2(y, oracle.linear_from_dequant(oracle.dequantize_weight(pp, pr, norms, seeds, cb, cb, 64), x.astype(np.float32))) < 4.9e-4
    lin.check_status()
    lin.close()


@pytest.mark.parametrize("outs", [(3584, 512, 512), (200, 3000), (64, 130, 9000, 64), (512, 512)])
@pytest.mark.parametrize("m", [9, 64, 300])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("cols", [1536, 4096])
def test_grouped_matrices_of_other_splits(tq, oracle, outs, m, shared, cols):
    """Matrices whose K is split differently (few weight rows: many splits), in any order, against calls of their own: the same bits."""
    import torch
    rng = np.random.default_rng(m + sum(outs))
    cb = oracle.codebook(4)[0]
    c = tq.codebook_from_centroids(cb)
    lins = []
    for o in outs:
        w = (rng.standard_normal((o, cols)) * 0.02).astype(np.float32)
        lins.append(tq.TurboQuantLinear(cols, o, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, 128, shared)), c, c, 128))
    x = torch.from_numpy(rng.standard_normal((m, cols)).astype(np.float16)).cuda()
    for lin, y in zip(lins, tq.forward_group(lins, x)):
        assert torch.equal(y, lin.forward(x))
        lin.check_status()
    for lin in lins:
        lin.close()


@pytest.mark.parametrize("m", [128, 256])
@pytest.mark.parametrize("shared", [True, False])
def test_weight_tiles_that_wait_for_their_slot(tq, m, shared):
    """Tall activation tiles: the products are slower than the lookups, so that every weight tile is written as soon as the MMAs have read the
    one before it in its slot.  Columns of one pipeline stage in 16 have an activation, the others' weights are a hundred times as large: a tile
    that is read too late or overwritten too early does not go unseen.  Against the dequantised weights; the tolerance of the tile edges."""
    import torch
    c = tq.generate_codebook(4)
    g = torch.Generator(device="cuda").manual_seed(m)
    cols, rows = 8192, 20000
    stage = torch.arange(cols, device="cuda") // 128
    some = (stage % 16 == 5).float()
    w = torch.randn((rows, cols), device="cuda", generator=g) * (2.0 - 1.98 * some)
    lin = tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, 128, shared)), c, c, 128)
    x = (torch.randn((m, cols), device="cuda", generator=g) * some).half()
    back = lin.dequantize(out=torch.empty((rows, cols), device="cuda", dtype=torch.float16))
    y = lin.forward(x)
    want = x.double() @ back.double().T
    assert rel_l2(y.cpu().numpy(), want.cpu().numpy()) < 4.9e-4 + 2.0 ** -11   # (and the dequantised weights' own rounding)
    for _ in range(10):
        assert torch.equal(lin.forward(x), y)
    lin.check_status()
    lin.close()
