"""The forward fused with an all-gather, for layers whose activation is rotated by a kernel of its own: blocks above 256 columns, two
rotations, several rows.  With flags to wait for, that kernel runs behind the wait."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def pointers(values):
    return (C.c_void_p * len(values))(*[int(v) for v in values])


@pytest.mark.parametrize("block,shared", [(512, True), (128, False), (512, False)], ids=["wide", "dual", "wide_dual"])
@pytest.mark.parametrize("batch", [1, 3, 8])
def test_all_gather_of_layers_rotated_in_front(tq, block, shared, batch):
    """Two ranks emulated on one stream: every flag that a call waits for has been raised by a call before it."""
    torch = pytest.importorskip("torch")
    L = tq.load()
    world, rows, cols = 2, 144, 1024
    total = world * rows
    g = torch.Generator(device="cuda").manual_seed(batch)
    c = tq.generate_codebook(4)
    lins = []
    for _ in range(world):
        w = torch.randn((rows, cols), generator=g, device="cuda") * 0.02
        lins.append(tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block))
    nbytes = batch * total * 2
    bufs = [torch.zeros(nbytes + 256, dtype=torch.uint8, device="cuda") for _ in range(world)]
    flags = [b.data_ptr() + nbytes for b in bufs]
    ex = [L.tq_exchange_create(r, world) for r in range(world)]
    x = torch.randn((batch, cols), generator=g, device="cuda").half()
    want = torch.cat([lin.forward(x) for lin in lins], dim=1)
    for step in range(3):
        for r in range(world):
            wait = C.c_void_p(flags[r]) if step > 0 else None   # nothing to wait for before the first exchange
            rc = L.tq_linear_forward_allgather(lins[r].handle, ex[r], C.c_void_p(x.data_ptr()), batch, pointers([bufs[r].data_ptr(), bufs[1 - r].data_ptr()]),
                                               world, total, r * rows, pointers(flags), world, wait, world, None)
            assert rc == 0, L.tq_last_error().decode()
        torch.cuda.synchronize()
        for r in range(world):
            assert torch.equal(bufs[r][:nbytes].view(torch.float16).view(batch, total), want), (step, r)
            assert bufs[r][nbytes:nbytes + 8].view(torch.int32).tolist() == [step + 1, step + 1]
        for b in bufs:
            b[:nbytes].zero_()
    for r in range(world):
        assert L.tq_exchange_wait(ex[r], C.c_void_p(flags[r]), world, None) == 0   # the last exchange
        assert L.tq_exchange_status(ex[r]) == 0
        lins[r].check_status()
        L.tq_exchange_free(ex[r])
        lins[r].close()


def waiting_layer(tq, torch, L, block, shared, batch):
    """A layer, its exchange, a gathered buffer with flags, and two flags to wait for in page-locked memory, not raised."""
    rows, cols = 144, 1024
    g = torch.Generator(device="cuda").manual_seed(batch + block)
    c = tq.generate_codebook(4)
    w = torch.randn((rows, cols), generator=g, device="cuda") * 0.02
    lin = tq.TurboQuantLinear(cols, rows, tq.quantize_weight(w, c, c, tq.QuantizerConfig(4, 4, block, shared)), c, c, block)
    ex = L.tq_exchange_create(0, 2)
    buf = torch.zeros(batch * 2 * rows * 2 + 256, dtype=torch.uint8, device="cuda")
    x, late = (torch.randn((batch, cols), generator=g, device="cuda").half() for _ in range(2))
    raised = torch.zeros(32, dtype=torch.int32).pin_memory()

    def forward():
        flags = buf.data_ptr() + batch * 2 * rows * 2
        return L.tq_linear_forward_allgather(lin.handle, ex, C.c_void_p(x.data_ptr()), batch, pointers([buf.data_ptr()]), 1, 2 * rows, 0,
                                             pointers([flags]), 1, C.c_void_p(raised.data_ptr()), 2, None)

    def result():
        return buf[:batch * 2 * rows * 2].view(torch.float16).view(batch, 2 * rows)[:, :rows]

    return lin, ex, x, late, raised, forward, result


@pytest.mark.parametrize("block,shared", [(512, True), (128, False), (512, False)], ids=["wide", "dual", "wide_dual"])
@pytest.mark.parametrize("batch", [1, 3, 8])
def test_the_rotation_reads_what_arrives_before_the_flags(tq, block, shared, batch):
    """The forward is queued while its flags are low; then the copy engine brings another activation, and the host raises the flags (well
    within the second that the kernel waits)."""
    torch = pytest.importorskip("torch")
    L = tq.load()
    lin, ex, x, late, raised, forward, result = waiting_layer(tq, torch, L, block, shared, batch)
    old, want = lin.forward(x), lin.forward(late)
    assert not torch.equal(old, want)
    arriving = late.cpu().pin_memory()
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert forward() == 0, L.tq_last_error().decode()
    with torch.cuda.stream(side):
        x.copy_(arriving, non_blocking=True)
    side.synchronize()
    raised.fill_(1)
    torch.cuda.synchronize()
    lin.check_status()
    assert torch.equal(result(), want)
    L.tq_exchange_free(ex)
    lin.close()


def test_flags_that_are_never_raised(tq):
    """The wait in front of the rotation ends after a second, with the status of a lost peer."""
    torch = pytest.importorskip("torch")
    L = tq.load()
    lin, ex, x, _, _, forward, _ = waiting_layer(tq, torch, L, 512, False, 3)
    torch.cuda.synchronize()
    assert forward() == 0, L.tq_last_error().decode()
    with pytest.raises(tq.TQError, match="peer wait"):
        lin.check_status()
    L.tq_exchange_free(ex)
    lin.close()
