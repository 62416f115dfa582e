"""The decoder glue at the sizes where its 16-byte accesses end: columns that are no multiple of 8, more columns than a CTA
keeps in registers, tensors that start 4 bytes off a 16-byte boundary, head sizes around the row kernel's.  fp16 outputs of
fp32 arithmetic: 2^-11 relative per value; the rotary angles carry fp32's 2^-24 times up to 4096 radians on top."""
import ctypes as C

import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 6e-4


def _at(torch, a, offset):
    """The array on the device, `offset` halves into an aligned buffer."""
    room = torch.empty(a.size + 8, dtype=torch.float16, device="cuda")
    t = room[offset:][: a.size].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("offset", [0, 2])
@pytest.mark.parametrize("rows,cols", [(1, 2), (3, 30), (2, 2048), (70, 3586), (2, 8192), (3, 9000)])
def test_sum_and_rmsnorm(tq, rows, cols, offset):
    import torch
    L = tq.load()
    rng = np.random.default_rng(rows + cols)
    slots = [rng.standard_normal((rows, cols)).astype(np.float16) for _ in range(2)]
    res, w = rng.standard_normal((rows, cols)).astype(np.float16), (1 + 0.1 * rng.standard_normal(cols)).astype(np.float16)
    both, resd, wd = _at(torch, np.stack(slots), offset), _at(torch, res, offset), _at(torch, w, offset)
    outs = [_at(torch, np.zeros((rows, cols), np.float16), offset) for _ in range(4)]
    n = rows * cols
    assert L.tq_exchange_sum_f16(_p(both), 2, n, n, _p(resd), _p(outs[0]), None) == 0
    assert L.tq_rmsnorm_f16(_p(outs[0]), _p(wd), _p(outs[1]), rows, cols, 1e-6, None) == 0
    assert L.tq_exchange_sum_f16_rmsnorm(_p(both), 2, n, rows, cols, _p(resd), _p(outs[2]), _p(wd), _p(outs[3]), 1e-6, None) == 0
    torch.cuda.synchronize()
    want = ((res.astype(np.float32) + slots[0].astype(np.float32)) + slots[1].astype(np.float32)).astype(np.float16)
    assert np.array_equal(outs[0].cpu().numpy(), want) and torch.equal(outs[2], outs[0]) and torch.equal(outs[3], outs[1])
    x = want.astype(np.float64)
    assert rel_l2(outs[1].cpu().numpy(), x / np.sqrt((x ** 2).mean(axis=1, keepdims=True) + 1e-6) * w.astype(np.float64)) < TOL


@pytest.mark.parametrize("offset", [0, 2])
@pytest.mark.parametrize("rows,inter", [(1, 2), (5, 1000), (3, 18944), (2, 2046)])
def test_swiglu(tq, rows, inter, offset):
    import torch
    rng = np.random.default_rng(inter)
    gu = (3 * rng.standard_normal((rows, 2 * inter))).astype(np.float16)
    d, act = _at(torch, gu, offset), _at(torch, np.zeros((rows, inter), np.float16), offset)
    assert tq.load().tq_swiglu_f16(_p(d), _p(act), rows, inter, None) == 0
    g, u = gu[:, :inter].astype(np.float64), gu[:, inter:].astype(np.float64)
    assert rel_l2(act.cpu().numpy(), g / (1 + np.exp(-g)) * u) < TOL


@pytest.mark.parametrize("offset", [0, 2])
@pytest.mark.parametrize("heads,kv_heads,dim", [(1, 1, 2), (3, 1, 16), (7, 2, 24), (28, 4, 128), (5, 5, 64), (2, 1, 512), (2, 1, 528)])
def test_rope(tq, heads, kv_heads, dim, offset):
    import torch
    rng = np.random.default_rng(dim + heads)
    pos = np.array([0, 1, 4095], np.int32)
    x = [rng.standard_normal((3, h, dim)).astype(np.float16) for h in (heads, kv_heads)]
    d = [_at(torch, a, offset) for a in x]
    pd = torch.from_numpy(pos).cuda()
    assert tq.load().tq_rope_qk_f16(_p(d[0]), _p(d[1]), _p(pd), 3, heads, kv_heads, dim, 1e6, None) == 0
    half = dim // 2
    ang = (pos[:, None].astype(np.float64) * 1e6 ** (-2.0 * np.arange(half) / dim))[:, None, :]
    for a, got in zip(x, d):
        lo, hi = a[..., :half].astype(np.float64), a[..., half:].astype(np.float64)
        want = np.concatenate([lo * np.cos(ang) - hi * np.sin(ang), hi * np.cos(ang) + lo * np.sin(ang)], axis=-1)
        assert rel_l2(got.cpu().numpy(), want) < TOL


@pytest.mark.parametrize("n_slots,residual", [(1, False), (1, True), (3, False), (3, True)])
@pytest.mark.parametrize("cols,offset", [(8, 0), (2056, 0), (16400, 0), (2056, 2)])
def test_sum_of_slots_and_rmsnorm(tq, n_slots, residual, cols, offset):
    """One CTA a row, with and without whole 16-byte pieces, against the sum and the norm on their own."""
    import torch
    L = tq.load()
    rng = np.random.default_rng(cols + n_slots)
    rows, n = 3, 3 * cols
    slots = _at(torch, rng.standard_normal((n_slots, rows, cols)).astype(np.float16), offset)
    res = _at(torch, rng.standard_normal((rows, cols)).astype(np.float16), offset) if residual else None
    w = _at(torch, (1 + 0.1 * rng.standard_normal(cols)).astype(np.float16), offset)
    outs = [_at(torch, np.zeros((rows, cols), np.float16), offset) for _ in range(4)]
    r = _p(res) if residual else None
    assert L.tq_exchange_sum_f16(_p(slots), n_slots, n, n, r, _p(outs[0]), None) == 0
    assert L.tq_rmsnorm_f16(_p(outs[0]), _p(w), _p(outs[1]), rows, cols, 1e-6, None) == 0
    assert L.tq_exchange_sum_f16_rmsnorm(_p(slots), n_slots, n, rows, cols, r, _p(outs[2]), _p(w), _p(outs[3]), 1e-6, None) == 0
    torch.cuda.synchronize()
    want = res.float() if residual else torch.zeros((rows, cols), device="cuda")
    for s in range(n_slots):
        want = want + slots[s].float()
    assert torch.equal(outs[0], want.half()) and torch.equal(outs[2], outs[0]) and torch.equal(outs[3], outs[1])


@pytest.mark.parametrize("n_slots,residual", [(1, True), (3, False), (8, True)])
@pytest.mark.parametrize("cols,offset", [(c, 0) for c in (2040, 2048, 2056, 4088, 4096, 4104, 8184, 8192, 8200)] + [(2046, 0), (8194, 0), (4096, 2)])
def test_rows_at_the_ends_of_what_stays_in_registers(tq, n_slots, residual, cols, offset):
    """One, two, four steps of 2048 columns in registers, and more: the norm against 64 bits, the fused form against the norm on its own."""
    import torch
    L = tq.load()
    rng = np.random.default_rng(cols + n_slots)
    rows, n = 5, 5 * cols
    slots = _at(torch, rng.standard_normal((n_slots, rows, cols)).astype(np.float16), offset)
    res = _at(torch, rng.standard_normal((rows, cols)).astype(np.float16), offset) if residual else None
    w = _at(torch, (1 + 0.1 * rng.standard_normal(cols)).astype(np.float16), offset)
    outs = [_at(torch, np.zeros((rows, cols), np.float16), offset) for _ in range(4)]
    r = _p(res) if residual else None
    assert L.tq_exchange_sum_f16(_p(slots), n_slots, n, n, r, _p(outs[0]), None) == 0
    assert L.tq_rmsnorm_f16(_p(outs[0]), _p(w), _p(outs[1]), rows, cols, 1e-6, None) == 0
    assert L.tq_exchange_sum_f16_rmsnorm(_p(slots), n_slots, n, rows, cols, r, _p(outs[2]), _p(w), _p(outs[3]), 1e-6, None) == 0
    torch.cuda.synchronize()
    want = res.float() if residual else torch.zeros((rows, cols), device="cuda")
    for s in range(n_slots):
        want = want + slots[s].float()
    assert torch.equal(outs[0], want.half()) and torch.equal(outs[2], outs[0]) and torch.equal(outs[3], outs[1])
    x = outs[0].double()
    assert rel_l2(outs[1].cpu().numpy(), (x / torch.sqrt((x ** 2).mean(1, keepdim=True) + 1e-6) * w.double()).cpu().numpy()) < TOL
