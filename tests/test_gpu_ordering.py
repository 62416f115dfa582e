"""Calls that read what the call before them wrote, with nothing in between, against the same calls with a wait behind each: the same bits.  Every kernel
here is launched before the one in front of it has ended and has to read behind its wait alone."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _layer(tq, g, cols, rows, block=128, shared=True):
    import torch
    c = tq.generate_codebook(4)
    w = torch.randn((rows, cols), generator=g, device="cuda") * cols ** -0.5
    return tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block)


def _same_without_waits(run):
    """run(stream, wait): a chain of calls whose results are returned.  In a graph, and queued one after the other behind a pass of other inputs' results."""
    import torch
    want = run(torch.cuda.current_stream(), torch.cuda.synchronize)
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        run(stream, lambda: None)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        got = run(stream, lambda: None)
    for _ in range(10):
        for t in got:
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    del graph


# one row to many, blocks of one, two and four chunks of 256 columns, one rotation and two
@pytest.mark.parametrize("block,shared", [(64, True), (128, True), (256, False), (512, True), (512, False), (1024, True)])
@pytest.mark.parametrize("m", [1, 3, 8, 9, 16, 33, 64, 100, 128, 129, 300])
def test_chain_of_linears(tq, m, block, shared):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    wide = [_layer(tq, g, 1024, 3072, block, shared) for _ in range(3)]
    down = _layer(tq, g, 3072, 1024, block, shared)
    long = _layer(tq, g, 1024, 19456, block, shared)      # more tiles than SMs
    back = _layer(tq, g, 19456, 1024, block, shared)
    x = torch.randn((m, 1024), generator=g, device="cuda").half()

    def run(stream, wait):
        y, out = x, []
        for _ in range(3):
            ys = tq.forward_group(wide, y, stream=stream)
            wait()
            y = ys[2]
            for layer in (down, long, back, wide[0], down):
                y = layer.forward(y, stream=stream)
                wait()
            out += [*ys, y]
        return out

    _same_without_waits(run)
    for layer in (*wide, down, long, back):
        layer.check_status()
        layer.close()


@pytest.mark.parametrize("rows,dim,block", [(1, 128, 128), (2, 64, 512), (8, 128, 512), (12, 128, 128), (70, 64, 512)])
def test_chain_of_a_decoder_layer(tq, rows, dim, block):
    """Norms, projections, rotary embedding, the KV append, attention over it, the values back, sums and SwiGLU."""
    import torch
    L, g = tq.load(), torch.Generator(device="cuda").manual_seed(rows + dim)
    heads, kv, hidden, inter = 512 // dim, 256 // dim, 512, 1024
    q, k, v = (_layer(tq, g, hidden, n * dim, block) for n in (heads, kv, kv))
    o, gate_up, down = _layer(tq, g, heads * dim, hidden, block), _layer(tq, g, hidden, 2 * inter, block), _layer(tq, g, inter, hidden, block)
    norm = torch.rand((hidden,), generator=g, device="cuda").half() + 0.5
    x = torch.randn((rows, hidden), generator=g, device="cuda").half()
    positions = torch.arange(rows, device="cuda", dtype=torch.int32)

    def p(t):
        return C.c_void_p(t.data_ptr())

    def run(stream, wait):
        st = C.c_void_p(stream.cuda_stream)
        new = lambda *shape: torch.empty(shape, device="cuda", dtype=torch.float16)   # noqa: E731
        check = tq._lib.check
        caches, h, out = [tq.TQKVCache(1, kv, dim) for _ in range(rows)], x, []
        for c in caches:
            c.reserve(0, 64)
        for _ in range(3):
            n = new(rows, hidden)
            check(L.tq_rmsnorm_f16(p(h), p(norm), p(n), rows, hidden, 1e-6, st), "rmsnorm")
            wait()
            qs, ks, vs = tq.forward_group([q, k, v], n, stream=stream)
            wait()
            check(L.tq_rope_qk_f16(p(qs), p(ks), p(positions), rows, heads, kv, dim, 1e6, st), "rope")
            wait()
            tq.append_batch(caches, 0, ks.view(rows, kv, dim), vs.view(rows, kv, dim), stream=stream)
            wait()
            a = tq.compressed_attention(caches, 0, qs.view(rows, heads, dim), use_qjl=True, stream=stream)
            wait()
            values = new(1, kv, dim)
            caches[-1].get_values_fp16(0, caches[-1].seq_length() - 1, caches[-1].seq_length(), out=values, stream=stream)
            wait()
            y = o.forward(a.view(rows, heads * dim), stream=stream)
            wait()
            s, n2 = new(rows, hidden), new(rows, hidden)
            check(L.tq_exchange_sum_f16_rmsnorm(p(y), 1, rows * hidden, rows, hidden, p(h), p(s), p(norm), p(n2), 1e-6, st), "sum")
            wait()
            gu, act = gate_up.forward(n2, stream=stream), new(rows, inter)
            wait()
            check(L.tq_swiglu_f16(p(gu), p(act), rows, inter, st), "swiglu")
            wait()
            d, h2 = down.forward(act, stream=stream), new(rows, hidden)
            wait()
            check(L.tq_exchange_sum_f16(p(d), 1, rows * hidden, rows * hidden, p(s), p(h2), st), "sum")
            wait()
            h = h2
            out += [qs, ks, vs, a, values, s, h]
        torch.cuda.synchronize()
        for c in caches:
            c.close()
        return out

    want = run(torch.cuda.current_stream(), torch.cuda.synchronize)
    for _ in range(5):
        torch.empty(1 << 24, device="cuda").fill_(float("nan"))   # (what is allocated next holds nothing of the pass before)
        torch.cuda.synchronize()
        busy = torch.randn((4096, 4096), device="cuda")
        busy = busy @ busy @ busy                                 # the calls queue up behind it
        assert all(torch.equal(a, b) for a, b in zip(run(torch.cuda.current_stream(), lambda: None), want))
    for layer in (q, k, v, o, gate_up, down):
        layer.close()
