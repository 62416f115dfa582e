"""Device memory kept between objects: what it must not make work, what it must give back."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

GROW_IN_CAPTURE = """
import torch
import turboquant_mlx_core_b200 as tq
side = torch.cuda.Stream()
kv = torch.randn((257, 2, 128), device="cuda").half()
torch.cuda.synchronize()
c = tq.TQKVCache(1, 2, 128)
c.append(0, kv[:256], kv[:256], stream=side)          # full: the next token doubles the storage
torch.cuda.synchronize()
before = c.get_keys_fp16(0, 0, 256)
other = tq.TQKVCache(1, 2, 128)
other.reserve(0, 512)                                 # leaves a block of the doubled size behind, nothing pending on it
other.append(0, kv[:1], kv[:1], stream=side)
torch.cuda.synchronize()
other.close()
what = None
try:
    with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=side):
        try:
            c.append(0, kv[256:], kv[256:], stream=side)
        except tq.TQError as e:
            what = e
except RuntimeError:
    pass                                              # the capture that the refusal ended
torch.cuda.synchronize()
assert what is not None, "growing inside a capture was not refused"
assert c.seq_length() == 256 and (c.get_keys_fp16(0, 0, 256).view("u2") == before.view("u2")).all()
c.append(0, kv[256:], kv[256:])
assert c.seq_length() == 257 and (c.get_keys_fp16(0, 0, 256).view("u2") == before.view("u2")).all()
print("ok")
"""


def test_storage_does_not_grow_inside_a_capture():
    """A kept block must not let an append inside a capture move the storage: the copy would run at replay, the host would
    count on it now.  In a process of its own, which the broken capture ends with."""
    r = subprocess.run([sys.executable, "-c", GROW_IN_CAPTURE], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr


def test_a_fit_needs_no_memory_that_is_not_there(tq):
    """With less free memory than a copy of the samples takes, the fit goes over the samples where they are."""
    torch = pytest.importorskip("torch")
    x = torch.randn((1 << 28,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    want = tq.generate_codebook_from_data(x, 4, 3)
    ones = tq.generate_codebook_from_data(torch.ones(100000, device="cuda"), 4, 3)   # the other path's kernels are loaded
    assert ones is not None
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    fill = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (768 << 20)), dtype=torch.uint8, device="cuda")
    try:
        got = tq.generate_codebook_from_data(x, 4, 3)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert np.all(np.abs(got.centroids - want.centroids) <= 3e-6 * np.abs(want.centroids) + 3e-7)


def test_kept_memory_goes_back_on_request(tq):
    torch = pytest.importorskip("torch")
    tq.release_cached_memory()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    kv = torch.zeros((4096, 2, 128), device="cuda", dtype=torch.float16)
    c = tq.TQKVCache(1, 2, 128)
    c.reserve(0, 400_000)                                   # about 100 MB
    c.append(0, kv, kv)
    c.close()                                               # kept, with the append still queued
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] < before - (64 << 20)
    assert tq.release_cached_memory() > (64 << 20)
    assert torch.cuda.mem_get_info()[0] > before - (32 << 20)
    assert tq.release_cached_memory() == 0


def test_an_idle_block_comes_before_a_pending_one(tq):
    """Storage that the host must be able to rely on at once does not wait for queued work while an idle block is there."""
    torch = pytest.importorskip("torch")
    tq.release_cached_memory()
    kv = torch.randn((4096, 2, 128), device="cuda").half()
    a = torch.randn((8192, 8192), device="cuda")
    side = torch.cuda.Stream()

    def make(stream=None):
        c = tq.TQKVCache(1, 2, 128)
        c.reserve(0, 4096, stream=stream)
        return c

    idle, pending = make(), make()
    idle.close()
    torch.cuda.synchronize()
    for _ in range(6):
        a = a @ a * 1e-4                                    # tens of milliseconds on the legacy stream
    pending.append(0, kv, kv)
    pending.close()
    end = torch.cuda.Event()
    end.record()
    c = make(side)                                          # (the call waits for its stream, on which nothing is queued)
    assert not end.query()
    c.append(0, kv, kv, stream=side)
    got = torch.empty((4096, 2, 128), dtype=torch.float16, device="cuda")
    c.get_keys_fp16(0, 0, 4096, out=got, stream=side)
    torch.cuda.synchronize()
    other = make()                                          # the pending one, by now done
    other.append(0, kv, kv)
    assert np.array_equal(other.get_keys_fp16(0, 0, 4096).view(np.uint16), got.cpu().numpy().view(np.uint16))
    c.close()
    other.close()
