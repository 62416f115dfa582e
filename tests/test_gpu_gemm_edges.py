"""The many-row linear at the edges of its tiles and of the tile loop: weight rows around the 16-row code tiles and the 128-row tile, activation
rows around the 16-row MMA step and the 256-row tile, every WHT block size, K blocks that do not fill a stage, one and two
rotations.  Tolerance: fp16 rounds the rotated activation, the table and the result by up to 2^-11 each, independently; the
root mean square of three such errors over a row is below 2^-11 * sqrt(3 / 3) = 4.9e-4."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

CASES = [
    # weight rows, columns, WHT block, activation rows, shared rotation
    (1, 64, 64, 9, True),
    (15, 192, 64, 16, True),
    (17, 320, 32, 17, False),
    (127, 256, 256, 31, True),
    (129, 512, 512, 33, False),
    (257, 1024, 1024, 255, True),
    (113, 1536, 512, 257, True),
    (96, 2048, 1024, 10, False),
    (200, 320, 64, 300, False),       # two rotations and full tiles: the shortest ring
    # more tiles than SMs: the ring runs on from tile to tile
    (57000, 64, 64, 20, True),        # one stage per tile, two accumulators in turn
    (19100, 192, 64, 257, False),     # ... one accumulator, an odd number of K blocks, a short last token tile
    (38000, 320, 64, 130, True),
]


@pytest.mark.parametrize("case", CASES, ids=[f"{c[0]}x{c[1]}_b{c[2]}_m{c[3]}_{'s' if c[4] else 'd'}" for c in CASES])
@pytest.mark.parametrize("aligned", [True, False], ids=["x16", "x2"])
def test_many_row_linear_at_tile_edges(tq, oracle, case, aligned):
    import torch
    rows, cols, bs, m, shared = case
    rng = np.random.default_rng(rows + cols + m)
    cb = oracle.codebook(4)[0]
    w = (rng.standard_normal((rows, cols)) * 0.02).astype(np.float16).astype(np.float32)
    pp, pr, norms, seeds = oracle.quantize_weight(w, cb, cb, 4, 4, bs, shared)
    want_w = oracle.dequantize_weight(pp, pr, norms, seeds, cb, cb, bs)
    xh = rng.standard_normal((m, cols)).astype(np.float16)
    c = tq.codebook_from_centroids(cb)
    lin = tq.TurboQuantLinear(cols, rows, tq.QuantizedWeight(pp, pr, norms, seeds), c, c, bs)
    room = torch.empty(m * cols + 8, dtype=torch.float16, device="cuda")
    x = room[(0 if aligned else 1):][: m * cols].view(m, cols)   # the rotation's 16-byte loads need an aligned activation
    x.copy_(torch.from_numpy(xh))
    y = lin.forward(x).cpu().numpy()
    want = oracle.linear_from_dequant(want_w, xh.astype(np.float32))
    assert rel_l2(y, want) < 4.9e-4
    assert rel_l2(lin.forward(x[:8]).cpu().numpy(), want[:8]) < 4.9e-4
    lin.check_status()
    lin.close()
