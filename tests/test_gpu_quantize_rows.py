"""The quantiser's row norms, codes and planes at the edges of their kernels: bit for bit the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))


# rows around the 32 of a CTA, columns around the 128 of a tile and the ring of four tiles; every block size
@pytest.mark.parametrize("rows,cols,block", [
    (1, 32, 32), (31, 96, 32), (32, 128, 128), (33, 160, 32), (65, 448, 64), (7, 640, 128), (40, 768, 256), (3, 1536, 512), (130, 1024, 1024),
])
@pytest.mark.parametrize("bits", [(4, 4, True), (4, 4, False), (5, 3, True), (3, 2, False)], ids=["shared", "dual", "five", "few"])
def test_quantised_rows_match_the_oracle(tq, oracle, rows, cols, block, bits):
    torch = pytest.importorskip("torch")
    pb, rb, shared = bits
    rng = np.random.default_rng(rows * cols)
    w = (rng.standard_normal((rows, cols)) * 0.02).astype(np.float32)
    w[0, ::5] = 0.0
    if rows > 2:
        w[1] = 0.0
        w[2] *= 1e4
    cp, cr = tq.generate_codebook(pb), tq.generate_codebook(rb)
    want = oracle.quantize_weight(w, cp.centroids, cr.centroids, pb, rb, block, shared)
    room = torch.zeros(rows * cols + 1, device="cuda")
    for at in (0, 1):   # weights on a 16-byte boundary, and not
        dev = room[at:at + rows * cols].view(rows, cols).copy_(torch.from_numpy(w))
        qw = tq.quantize_weight(dev, cp, cr, tq.QuantizerConfig(pb, rb, block, shared))
        assert same(qw.packed_primary, want[0]) and same(qw.packed_residual, want[1])
        assert same(qw.norms, want[2]) and same(qw.seeds, want[3])


def test_codebooks_that_do_not_ascend(tq):
    """A code is the number of boundaries below the value, whatever their order."""
    rng = np.random.default_rng(3)
    w = (rng.standard_normal((20, 256)) * 0.02).astype(np.float32)
    c = tq.generate_codebook(4)
    down = tq.codebook_from_centroids(c.centroids[::-1].copy())
    cfg = tq.QuantizerConfig(4, 0, 128, False)
    assert same(tq.quantize_weight(w, down, c, cfg).packed_primary, tq.quantize_weight(w, c, c, cfg).packed_primary)
