"""One activation row of a host caller as a parameter of the decode kernel, at the sizes where the parameter block or the way of the
row changes: against the same row in device memory, the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,block", [(64, 64), (2048, 128), (2112, 64), (4096, 256), (4160, 64), (8192, 32), (8256, 64), (15872, 256), (15936, 32),
                                        (4096, 512)])
@pytest.mark.parametrize("shared", [True, False])
def test_host_row_sizes(tq, n_in, block, shared):
    import torch
    c = tq.generate_codebook(4)
    g = torch.Generator(device="cuda").manual_seed(n_in)
    w = torch.randn((300, n_in), device="cuda", generator=g) * 0.02
    lin = tq.TurboQuantLinear(n_in, 300, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block)
    room = np.random.default_rng(n_in).standard_normal(n_in + 1).astype(np.float32)
    for x in (room[:n_in], room[1:], room[:n_in].astype(np.float16), np.where(np.arange(n_in) == 5, np.float32(1e6), room[:n_in])):
        got = lin.forward(x[None])
        with np.errstate(over="ignore"):
            want = lin.forward(torch.from_numpy(x[None].astype(np.float16)).cuda()).cpu().numpy()
        assert got.shape == (1, 300) and np.array_equal(got, want, equal_nan=True)
    lin.check_status()
    lin.close()
