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


@pytest.mark.parametrize("rows,n_out", [(1, 16384), (1, 16385), (2, 4096), (2, 4097), (8, 1024), (8, 1040), (9, 40)])   # stored by the kernel, and copied
def test_host_results_equal_device_results(tq, rows, n_out):
    torch = pytest.importorskip("torch")
    lin = make_linear(tq, 64, n_out)
    x = np.random.default_rng(n_out).standard_normal((rows, 64)).astype(np.float16)
    want = lin.forward(torch.from_numpy(x).cuda()).cpu().numpy()
    for _ in range(2):
        assert np.array_equal(lin.forward(x).view(np.uint16), want.view(np.uint16))
    lin.close()


@pytest.mark.parametrize("at", [0, 5, 63])
@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf, -np.inf, 65519.99, 65520.0, -65520.0, 2.0 ** -25, -2.98e-8, 1e-45])
def test_host_rounding_of_special_values(tq, at, value):
    """Rows of 64: eight values at a time, and a NaN among them."""
    torch = pytest.importorskip("torch")
    lin = make_linear(tq, 64, 16)
    x = np.random.default_rng(at).standard_normal((1, 64)).astype(np.float32)
    x[0, at] = value
    if np.isnan(value):
        x.view(np.uint32)[0, at] = 0x7f800001 if np.signbit(value) else 0xffc12345      # signalling, and with a payload
    got = lin.forward(x)
    want = lin.forward(torch.from_numpy(x).cuda())
    assert np.array_equal(got.view(np.uint16), want.cpu().numpy().view(np.uint16))
    lin.close()


@pytest.mark.parametrize("rows,n_in", [(1, 4096), (2, 4160), (5, 3200)])   # parameters and staging, as pageable rows
@pytest.mark.parametrize("dtype", ["float16", "float32"])
def test_page_locked_rows_are_read_in_stream_order(tq, rows, n_in, dtype):
    """Work queued on the stream writes the page-locked rows: the forward that follows sees what it wrote."""
    torch = pytest.importorskip("torch")
    lin = make_linear(tq, n_in, 80)
    x = torch.randn((rows, n_in), device="cuda").to(getattr(torch, dtype))
    want = lin.forward(x)
    a = torch.randn((8192, 8192), device="cuda")
    pinned = torch.zeros((rows, n_in), dtype=x.dtype).pin_memory()
    got = torch.empty_like(want)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for stream in (torch.cuda.default_stream(), side):
        pinned.zero_()
        with torch.cuda.stream(stream):
            for _ in range(4):
                a = a @ a * 1e-4                       # tens of milliseconds
            pinned.copy_(x, non_blocking=True)
            lin.forward(pinned, out=got, stream=stream)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    lin.close()


@pytest.mark.parametrize("dtype", ["float16", "float32"])
def test_a_captured_forward_reads_page_locked_rows_on_every_replay(tq, dtype):
    torch = pytest.importorskip("torch")
    lin = make_linear(tq, 1024, 80)
    x = [torch.randn((3, 1024), device="cuda").to(getattr(torch, dtype)) for _ in range(3)]
    want = [lin.forward(t) for t in x]
    pinned = torch.zeros((3, 1024), dtype=x[0].dtype).pin_memory()
    got = torch.empty_like(want[0])
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        lin.forward(pinned, out=got, stream=side)      # allocates what the capture must not
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        lin.forward(pinned, out=got, stream=side)
    for t, w in zip(x, want):
        pinned.copy_(t)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, w)
    del graph
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
