"""Large copies between the device and host memory, in pieces: whatever their number, with a short last piece, several at once, and
from several threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# bytes of the fp32 result around the bounds of 8 and 32 MB and of a piece; rows that end inside a piece
@pytest.mark.parametrize("rows,cols", [(64, 64), (2047, 1024), (2048, 1024), (2049, 1024), (8192, 1024), (8193, 1088), (20011, 1024)])
def test_host_results_equal_device_results(tq, rows, cols):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = torch.randn((rows, cols), generator=g, device="cuda") * 0.02
    c = tq.generate_codebook(4)
    cfg = tq.QuantizerConfig(4, 4, 64, True)
    device, host = tq.quantize_weight(w, c, c, cfg), tq.quantize_weight(w.cpu().numpy(), c, c, cfg)
    for name in ("packed_primary", "packed_residual", "norms", "seeds"):
        assert np.array_equal(getattr(device, name), getattr(host, name)), name
    lin = tq.TurboQuantLinear(cols, rows, host, c, c, 64)
    back = torch.empty((rows, cols), device="cuda")
    lin.dequantize(out=back)
    assert np.array_equal(lin.dequantize(np.float32).view(np.uint32), back.cpu().numpy().view(np.uint32))
    lin.close()


def test_five_bit_and_primary_only_planes_are_written_whole(tq, oracle):
    rng = np.random.default_rng(1)
    w = (rng.standard_normal((48, 256)) * 0.02).astype(np.float32)
    cb5, cb3 = tq.generate_codebook(5), tq.generate_codebook(3)
    for bits, res, shared in ((5, 3, True), (4, 0, False), (5, 0, False)):
        cb = cb5 if bits == 5 else tq.generate_codebook(4)
        for _ in range(3):   # (memory that held something else before)
            junk = np.full((48, 256), 0xA5, np.uint8)
            del junk
            qw = tq.quantize_weight(w, cb, cb3, tq.QuantizerConfig(bits, res, 128, shared))
            pp, pr, norms, _ = oracle.quantize_weight(w, cb.centroids, cb3.centroids, bits, res, 128, shared)
            assert np.array_equal(qw.packed_primary, pp) and np.array_equal(qw.packed_residual, pr)
            assert np.array_equal(qw.norms.view(np.uint32), norms.view(np.uint32))


def test_copies_from_several_threads(tq):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(2)
    c = tq.generate_codebook(4)
    weights = [torch.randn((3000, 1024), generator=g, device="cuda") * 0.02 for _ in range(4)]
    layers = [tq.TurboQuantLinear(1024, 3000, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, 128, True)), c, c, 128) for w in weights]
    alone = [lin.dequantize(np.float32) for lin in layers]
    got = [None] * 4

    def run(i):
        for _ in range(3):
            got[i] = layers[i].dequantize(np.float32)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(alone, got))


@pytest.mark.parametrize("kind", ["per_thread", "non_blocking"])
def test_host_weights_on_other_streams(tq, kind):
    """Weights of more than 32 MB in host memory, on a stream whose handle means another stream in every thread (cudaStreamPerThread = 2)
    and on one that does not wait for the default stream: the bits of device weights, call after call and beside a second thread."""
    torch = pytest.importorskip("torch")
    L = tq.load()
    c = tq.generate_codebook(4)
    cb = np.ascontiguousarray(c.centroids, np.float32)
    cols = 1024

    def quantize(w, rows, stream):
        planes = [np.empty((rows, cols // 2), np.uint8) for _ in range(2)]
        norms, seeds = np.empty(rows, np.float32), np.zeros(3, np.uint32)
        p = w.ctypes.data if isinstance(w, np.ndarray) else w.data_ptr()
        rc = L.tq_quantize_weight(p, rows, cols, cb.ctypes.data, cb.size, cb.ctypes.data, cb.size, 4, 4, 64, 1, planes[0].ctypes.data,
                                  planes[1].ctypes.data, norms.ctypes.data, seeds.ctypes.data, stream)
        assert rc == 0, L.tq_last_error().decode()
        return planes + [norms.view(np.uint32), seeds]

    def fit(w, stream):
        return [x for b in tq.fit_layer_codebooks(w, 64, 4, 4, 10, stream=stream) for x in (b.centroids, b.boundaries)]

    failures = []

    def work(rows):
        stream = 2 if kind == "per_thread" else torch.cuda.Stream().cuda_stream
        g = torch.Generator(device="cuda").manual_seed(rows)
        for _ in range(3):   # other weights each time: what an earlier call left in the staging is wrong
            w = torch.randn((rows, cols), generator=g, device="cuda") * 0.02
            torch.cuda.synchronize()
            host = w.cpu().numpy()
            for want, got in ((quantize(w, rows, None), quantize(host, rows, stream)), (fit(w, None), fit(host, stream))):
                failures.extend((rows, i) for i, (a, b) in enumerate(zip(want, got)) if not np.array_equal(a, b))

    threads = [threading.Thread(target=work, args=(rows,)) for rows in (8449, 20480)]   # 34.6 and 83.9 MB
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures


def test_page_locked_values_are_read_in_stream_order(tq):
    """Codebooks and seeds in page-locked memory that work queued on the default stream still writes."""
    torch = pytest.importorskip("torch")
    L = tq.load()
    rows, cols, block = 64, 256, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    w = torch.randn((rows, cols), generator=g, device="cuda") * 0.02
    c = tq.generate_codebook(4)
    cb = np.ascontiguousarray(c.centroids, np.float32)
    want = tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, False))

    def queued(values):
        """Page-locked memory that holds other values until a copy behind some milliseconds of work has run."""
        late = torch.full(values.shape, 1, dtype=values.dtype).pin_memory()
        on_device = values.cuda()
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)
        late.copy_(on_device, non_blocking=True)
        return late

    planes = [np.empty((rows, cols // 2), np.uint8) for _ in range(2)]
    norms, seeds = np.empty(rows, np.float32), np.zeros(3, np.uint32)
    late = queued(torch.from_numpy(cb))
    rc = L.tq_quantize_weight(w.data_ptr(), rows, cols, late.data_ptr(), cb.size, late.data_ptr(), cb.size, 4, 4, block, 0, planes[0].ctypes.data,
                              planes[1].ctypes.data, norms.ctypes.data, seeds.ctypes.data, None)
    assert rc == 0, L.tq_last_error().decode()
    assert np.array_equal(planes[0], want.packed_primary) and np.array_equal(planes[1], want.packed_residual)
    assert np.array_equal(norms, want.norms) and np.array_equal(seeds, want.seeds)

    layer = tq.TurboQuantLinear(cols, rows, want, c, c, block)
    late = queued(torch.from_numpy(want.seeds.view(np.int32)))
    h = L.tq_linear_create(cols, rows, want.packed_primary.ctypes.data, cols // 2, want.packed_residual.ctypes.data, want.norms.ctypes.data,
                           late.data_ptr(), cb.ctypes.data, cb.size, cb.ctypes.data, cb.size, block)
    assert h, L.tq_last_error().decode()
    back = torch.empty((rows, cols), device="cuda")
    assert L.tq_linear_dequantize(h, back.data_ptr(), 0, None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(back.cpu().numpy(), layer.dequantize(np.float32))
    L.tq_linear_free(h)
    layer.close()
