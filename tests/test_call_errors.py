"""Calls of the Python layer that are refused before any device work: the error's type is part of the interface."""
import numpy as np
import pytest

import turboquant_mlx_core_b200 as tq


def rows(n):
    return np.zeros((n, 2, 128), np.float16)


def test_no_caches():
    with pytest.raises(tq.TQError):
        tq.append_batch([], 0, rows(0), rows(0))
    with pytest.raises(ValueError):
        tq.append_batch([], 0, rows(1), rows(1))
    with pytest.raises(ValueError):
        tq.compressed_attention([], 0, rows(1))


@pytest.mark.parametrize("columns,block,what", [(34, 32, "divisible"), (66, 64, "divisible"), (48, 48, "power of two"), (64, 16, "power of two")])
def test_layer_fits_of_odd_shapes(columns, block, what):
    """The reason is the shape's, whatever the kernels in front of it want."""
    with pytest.raises(tq.TQError, match=what):
        tq.fit_layer_codebooks(np.ones((4, columns), np.float32), block)


@pytest.mark.gpu
def test_host_rows_where_device_rows_are_needed():
    torch = pytest.importorskip("torch")
    c = tq.TQKVCache(1, 2, 128)
    d = torch.zeros((1, 2, 128), dtype=torch.float16, device="cuda")
    for keys, values in ((d, rows(1)), (rows(1), d), (rows(1), rows(1))):
        with pytest.raises(tq.TQError):
            tq.append_batch([c], 0, keys, values)
    assert c.seq_length() == 0
    c.close()
    cb = tq.generate_codebook(4)
    qw = tq.quantize_weight(np.ones((16, 64), np.float32), cb, cb, tq.QuantizerConfig(4, 4, 64, True))
    lin = tq.TurboQuantLinear(64, 16, qw, cb, cb, 64)
    with pytest.raises(tq.TQError):
        tq.forward_group([lin, lin], np.zeros((2, 64), np.float16))
    lin.close()
