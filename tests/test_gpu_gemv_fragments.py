"""The decode kernel's activation in the order of its fragments: every padded number of rows, columns that end inside a 64-column block (two groups of
16 columns instead of four) and inside a warp's 256, blocks of one, two and four chunks, several chunks of columns, one rotation and two, rows
that are not 16-byte aligned.  Tolerance: TF32 (or as many bits of fp16) rounds the rotated activation and the table by up to 2^-11 each and the
result is rounded to fp16: three independent roundings, 2^-11 * sqrt(3 / 3)."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols,block", [(32, 32), (96, 32), (160, 32), (288, 32), (320, 64), (512, 512), (1024, 1024), (1536, 512), (4064, 32), (4128, 32),
                                        (5120, 128), (9216, 512), (10240, 1024)])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("aligned", [True, False], ids=["x16", "x2"])
def test_rows_and_columns_of_the_fragments(tq, oracle, cols, block, m, shared, aligned):
    import torch
    rows = 70
    rng = np.random.default_rng(cols + m)
    cb = oracle.codebook(4)[0]
    w = (rng.standard_normal((rows, cols)) * 0.02).astype(np.float16).astype(np.float32)
    pp, pr, norms, seeds = oracle.quantize_weight(w, cb, cb, 4, 4, block, shared)
    xh = rng.standard_normal((m, cols)).astype(np.float16)
    c = tq.codebook_from_centroids(cb)
    lin, other = (tq.TurboQuantLinear(cols, rows, tq.QuantizedWeight(pp, pr, norms, seeds), c, c, block) for _ in range(2))
    room = torch.empty(m * cols + 8, dtype=torch.float16, device="cuda")
    x = room[(0 if aligned else 1):][: m * cols].view(m, cols)
    x.copy_(torch.from_numpy(xh))
    want = oracle.linear_from_dequant(oracle.dequantize_weight(pp, pr, norms, seeds, cb, cb, block), xh.astype(np.float32))
    y = lin.forward(x)
    assert rel_l2(y.cpu().numpy(), want) < 4.9e-4
    for of_group in tq.forward_group([lin, other], x):
        assert torch.equal(of_group, y)
    lin.check_status()
    lin.close()
    other.close()
