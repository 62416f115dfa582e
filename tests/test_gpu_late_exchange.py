"""Linears directly behind a wait for another rank that is late, longer than the linears' own time limits (0.2 s) and shorter than the wait's (1 s): no error, and
the bits of the same calls without a wait.  The other rank is the host here: it copies the flag, or the packets, while the wait runs."""
import ctypes as C
import time

import pytest

pytestmark = pytest.mark.gpu

LATE = 0.45


def _layer(tq, g, cols, rows, shared=True):
    import torch
    c = tq.generate_codebook(4)
    w = torch.randn((rows, cols), generator=g, device="cuda") * cols ** -0.5
    return tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, 128, shared)), c, c, 128)


class _Late:
    """Rank 0 of two: wait() queues a wait for rank 1, arrive() is rank 1."""

    def __init__(self, tq, kind, g):
        import torch
        self.tq, self.L, self.kind = tq, tq.load(), kind
        self.ex = self.L.tq_exchange_create(0, 2)
        self.side = torch.cuda.Stream()
        if kind == "flags":
            self.words = torch.zeros(32, dtype=torch.int32, device="cuda")
            self.arrived = torch.ones(32, dtype=torch.int32).pin_memory()
            return
        rows, cols = 208, 512
        self.rows, n = rows, rows // 4
        self.bufs = [torch.zeros((2, 2, n, 4), dtype=torch.int32, device="cuda") for _ in range(2)]   # [epoch parity][source rank][packets]
        self.words = self.bufs[0][1, 1]
        self.arrived = torch.ones((n, 4), dtype=torch.int32).pin_memory()                             # (epoch 1 beside some halves)
        self.gathered = torch.zeros((1, 2 * rows), dtype=torch.float16, device="cuda")
        self.norm, self.normed = torch.ones(rows, dtype=torch.float16, device="cuda"), torch.empty(rows, dtype=torch.float16, device="cuda")
        sender, x = _layer(tq, g, cols, rows), torch.randn((1, cols), generator=g, device="cuda").half()
        assert self.L.tq_linear_forward_allgather_packets(sender.handle, self.ex, C.c_void_p(x.data_ptr()), 1, C.c_void_p(self.gathered.data_ptr()), 2 * rows,
                                                          (C.c_void_p * 2)(*(b.data_ptr() for b in self.bufs)), 0, None) == 0
        torch.cuda.synchronize()
        sender.close()

    def wait(self, stream):
        st, words = C.c_void_p(stream.cuda_stream), C.c_void_p(self.words.data_ptr())
        if self.kind == "flags":
            assert self.L.tq_exchange_wait(self.ex, words, 1, st) == 0
            return
        base, row = C.c_void_p(self.bufs[0].data_ptr()), C.c_void_p(self.gathered.data_ptr())
        if self.kind == "packets":
            assert self.L.tq_exchange_wait_packets(self.ex, base, self.rows, 1, row, 2 * self.rows, st) == 0
        elif self.kind == "sums":
            assert self.L.tq_exchange_sum_packets(self.ex, base, row, self.rows, None, row, st) == 0
        else:
            assert self.L.tq_exchange_sum_packets_rmsnorm(self.ex, base, row, 1, self.rows, None, row, C.c_void_p(self.norm.data_ptr()),
                                                            C.c_void_p(self.normed.data_ptr()), 1e-6, st) == 0

    def arrive(self):
        import torch
        with torch.cuda.stream(self.side):
            self.words.copy_(self.arrived, non_blocking=True)

    def close(self):
        assert self.L.tq_exchange_status(self.ex) == 0
        self.L.tq_exchange_free(self.ex)


# two groups of producers, one group (more CTAs than SMs), three; more stages than the ring has and fewer
@pytest.mark.parametrize("m,cols,outs,shared,kind", [(16, 1024, (3072,), True, "flags"), (64, 4096, (4096,), True, "flags"), (40, 2048, (2048,), False, "flags"),
                                                     (16, 3584, (3584, 512, 512), True, "flags"), (100, 3584, (3584, 512, 512), False, "flags"),
                                                     (32, 5120, (20480,), True, "flags"), (16, 4096, (4096,), True, "packets"), (16, 4096, (4096,), True, "sums"),
                                                     (16, 4096, (4096,), True, "sums+norm")])
def test_linear_behind_a_late_rank(tq, m, cols, outs, shared, kind):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + cols)
    layers = [_layer(tq, g, cols, out, shared) for out in outs]
    back = _layer(tq, g, outs[0], cols, shared)
    x = torch.randn((m, cols), generator=g, device="cuda").half()
    stream = torch.cuda.Stream()

    def calls():
        ys = tq.forward_group(layers, x, stream=stream) if len(layers) > 1 else [layers[0].forward(x, stream=stream)]
        return [*ys, back.forward(ys[0], stream=stream)]      # (its kernels are let come by the first call's)

    want = calls()
    torch.cuda.synchronize()
    late = _Late(tq, kind, g)
    late.wait(stream)
    got = calls()
    time.sleep(LATE)
    assert not stream.query()
    late.arrive()
    torch.cuda.synchronize()
    for layer in (*layers, back):
        layer.check_status()
        layer.close()
    late.close()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
