"""Activation rows in host memory: kernel parameters up to 31 744 bytes of fp16, page-locked staging above, pageable copies
for the largest; and storage that comes back from the memory pool.  The path moves the rows and rounds fp32 to fp16 (nearest
even), so the result equals the same call on device tensors bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make_linear(tq, n_in, n_out, seed=0):
    w = (np.random.default_rng(seed).standard_normal((n_out, n_in)) * 0.02).astype(np.float32)
    cb = tq.generate_codebook(4)
    qw = tq.quantize_weight(w, cb, cb, tq.QuantizerConfig(4, 4, 64, True))
    return tq.TurboQuantLinear(n_in, n_out, qw, cb, cb, 64)


# 64: one 128-byte row; 1024 / 4096: the parameter sizes' edges; 5 x 3136: just below, 5 x 3200: just above the largest;
# 9 rows: the GEMM; 2112 x 1024: more than the staging takes
@pytest.mark.parametrize("rows,n_in", [(1, 64), (1, 1024), (1, 1088), (1, 4096), (2, 4160), (5, 3136), (5, 3200), (9, 1024), (2112, 1024)])
@pytest.mark.parametrize("dtype", [np.float32, np.float16])
def test_host_rows_equal_device_rows(tq, rows, n_in, dtype):
    torch = pytest.importorskip("torch")
    lin = make_linear(tq, n_in, 80)
    x = np.random.default_rng(rows * n_in).standard_normal((rows, n_in)).astype(np.float32)
    x[0, :8] = [0.0, -0.0, 6.1e-5, 3.0e-6, 2.9e-8, 1.00048828125, -1.0014648438, 65504.0 * 1e-4]   # subnormals and ties
    x = x.astype(dtype)
    got = lin.forward(x)
    want = lin.forward(torch.from_numpy(x).cuda())
    assert np.array_equal(got.view(np.uint16), want.cpu().numpy().view(np.uint16))
    y = torch.empty((rows, 80), dtype=torch.float16, device="cuda")      # host rows, device result
    lin.forward(x, out=y)
    assert torch.equal(y, want)
    lin.close()


def test_a_recycled_cache_waits_for_its_predecessor(tq):
    """Storage released with work still queued is reused behind that work, on the same stream and on another one."""
    torch = pytest.importorskip("torch")
    heads, dim, n = 2, 128, 4096
    g = torch.Generator(device="cuda").manual_seed(1)
    kv = [torch.randn((n, heads, dim), generator=g, device="cuda").half() for _ in range(4)]
    want = []
    for t in kv:
        c = tq.TQKVCache(1, heads, dim)
        c.append(0, t, t)
        want.append(torch.from_numpy(c.get_keys_fp16(0, 0, n)))
        c.close()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for stream in (None, side):
        got = []
        for t in kv:
            c = tq.TQKVCache(1, heads, dim)
            c.append(0, t, t, stream=stream)
            out = torch.empty((n, heads, dim), dtype=torch.float16, device="cuda")
            c.get_keys_fp16(0, 0, n, out=out, stream=stream)
            c.close()
            got.append(out)
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a.cpu(), b)
