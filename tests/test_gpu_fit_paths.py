"""The two ways of the codebook fit: bucketed samples, and passes over all samples for data that repeats itself.  Centroids
within the rounding of a mean (one part in 2^24, taken a few times over: the tolerance of tests/test_codebook_fit.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 8193, 65537, 1_000_003])
@pytest.mark.parametrize("kind", ["scaled", "outliers", "1e9", "1e12", "-1e15", "lowest", "wide", "one value", "few values", "zeros"])
def test_fit_against_the_checker(tq, oracle, n, kind):
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n)
    if kind == "scaled":                # far from the codebook it starts from
        x = x * 1e-3 + 5e-4
    elif kind == "outliers":            # other bins' values must not enter a bin's sum
        x[:: max(1, n // 7)] *= 1e6
    elif kind in ("1e9", "1e12", "-1e15"):
        x[n // 2] = float(kind)
    elif kind == "lowest":              # masked samples
        x[:: max(1, n // 5)] = np.finfo(np.float32).min
    elif kind == "wide":                # 60 decades, and buckets of several exponents in a group
        x = x * 10.0 ** rng.uniform(-30, 30, n)
    elif kind == "one value":
        x[:] = 0.37
    elif kind == "few values":          # more of each than a bucket may hold (from 65537 on)
        x = np.array([-1.2, 0.1, 0.9])[rng.integers(0, 3, n)]
    else:
        x[: n // 2] = 0.0
    x = x.astype(np.float32)
    want, _ = oracle.fit_codebook(x, 4, 20)
    got = tq.generate_codebook_from_data(x, 4, 20)
    tol = 3e-6 * np.abs(want) + 3e-7
    assert np.all(np.abs(got.centroids - want) <= tol), np.abs(got.centroids - want).max()


def _keys(x):
    """The order-preserving keys that the buckets are the upper bits of."""
    u = x.view(np.uint32)
    return u ^ np.where(u >> 31 != 0, np.uint32(0xffffffff), np.uint32(0x80000000))


def _key_bits(n):
    return 9 + min(12, max(3, (n - 1).bit_length() - 13))


SOME = [[k] for k in range(8)] + [[3, 4], [2, 5], [0, 3, 4, 6], [1, 2, 5, 7], list(range(8))]


@pytest.mark.parametrize("n,eighths", [(n, e) for n in (3000, 300_000, 4_300_000) for e in SOME]
                         + [(n, e) for n in (1_500_000, 2_100_000) for e in ([3], [4], [0], [2, 5], [0, 3, 4, 6], list(range(8)))] + [(17_000_000, [0, 3, 4, 6])])
def test_samples_in_some_eighths_of_the_bucket_keys(tq, oracle, n, eighths):
    """A block of the bucket sums looks at one to eight ranges of buckets (1.5 M samples two, 2.1 M four, 4.3 M eight), evenly spread over the keys: with
    and without samples in one block.  Magnitudes from 1e-38 to 1e38, so the tolerance is that of a mean alone: nothing absolute hides
    the small ones, each of which has a case of its own."""
    rng = np.random.default_rng(n)
    e = rng.choice(eighths, n)                                   # sign and two bits of the exponent, in the order of the keys
    exponent = (np.where(e >= 4, e - 4, 3 - e) * 64 + rng.integers(1, 60, n)).astype(np.uint32)
    bits = (exponent << 23) | rng.integers(0, 1 << 23, n).astype(np.uint32) | np.where(e < 4, np.uint32(1) << 31, 0).astype(np.uint32)
    x = bits.view(np.float32)
    assert sorted(set((_keys(x) >> 29).tolist())) == sorted(eighths)
    want, _ = oracle.fit_codebook(x, 4, 6)
    got = tq.generate_codebook_from_data(x, 4, 6)
    assert np.all(np.abs(got.centroids - want) <= 3e-6 * np.abs(want)), (got.centroids, want)


@pytest.mark.parametrize("n", [255, 256, 257, 511, 512, 513, 767, 768, 769, 1023, 1024, 1025, 1280, 1281, 2304, 2305, 8192])
def test_a_boundary_in_a_bucket_of_this_many_samples(tq, oracle, n):
    """The iterations read a bucket in steps of 512 and of 256 values; all samples lie in one bucket, and so does a boundary."""
    x = np.random.default_rng(n).uniform(0.94, 0.995, n).astype(np.float32)
    assert len(np.unique(_keys(x) >> (32 - _key_bits(n)))) == 1
    want, _ = oracle.fit_codebook(x, 2, 20)
    boundary = (want[2] + want[3]) / 2
    assert x.min() < boundary < x.max()                          # (the samples are what the test takes them for)
    got = tq.generate_codebook_from_data(x, 2, 20)
    tol = 3e-6 * np.abs(want) + 3e-7
    assert np.all(np.abs(got.centroids - want) <= tol), np.abs(got.centroids - want).max()


@pytest.mark.parametrize("n", [200_000, 1_000_003])
@pytest.mark.parametrize("share", [0.05, 0.3, 1.0])
def test_crowded_samples_are_fitted_in_passes_over_all(tq, oracle, n, share):
    """One value in so many places that its bucket is not worth filling: seen beforehand, or when a boundary comes to it."""
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n).astype(np.float32)
    x[rng.random(n) < share] = 0.0
    want, _ = oracle.fit_codebook(x, 4, 20)
    got, again = (tq.generate_codebook_from_data(x, 4, 20) for _ in range(2))
    assert np.all(np.abs(got.centroids - want) <= 3e-6 * np.abs(want) + 3e-7)
    assert np.array_equal(got.centroids.view(np.uint32), again.centroids.view(np.uint32))


@pytest.mark.parametrize("kind", ["normal", "wide", "small", "one sign", "two magnitudes"])
def test_fit_counts_outside_of_the_window(tq, oracle, kind):
    """The counters on the SM hold 32 exponents at most: samples below them, of one sign, and nowhere near the codebook."""
    n = 2_200_003
    rng = np.random.default_rng(7)
    x = rng.standard_normal(n)
    if kind == "wide":
        x = x * 10.0 ** rng.uniform(-30, 30, n)
    elif kind == "small":
        x = x * 1e-39                       # subnormal numbers
    elif kind == "one sign":
        x = -np.abs(x)
    elif kind == "two magnitudes":
        x[: n // 2] *= 1e-20
        rng.shuffle(x)
    x = x.astype(np.float32)
    want, _ = oracle.fit_codebook(x, 4, 3)
    got, again = (tq.generate_codebook_from_data(x, 4, 3) for _ in range(2))
    assert np.all(np.abs(got.centroids - want) <= 3e-6 * np.abs(want) + 3e-7)
    assert np.array_equal(got.centroids.view(np.uint32), again.centroids.view(np.uint32))


@pytest.mark.parametrize("rows,cols,block", [(40, 64, 64), (300, 512, 512), (1024, 2048, 128)])
def test_layer_fits_side_by_side(tq, rows, cols, block):
    """The two fits of a layer in one launch: each as it is alone."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = torch.randn((rows, cols), generator=g, device="cuda") * 0.02
    both = tq.fit_layer_codebooks(w, block, 4, 3, 40)
    alone, _ = tq.fit_layer_codebooks(w, block, 4, 0, 40)
    assert np.array_equal(both[0].centroids.view(np.uint32), alone.centroids.view(np.uint32))
    host = tq.fit_layer_codebooks(w.cpu().numpy(), block, 4, 3, 40)
    assert all(np.array_equal(a.centroids.view(np.uint32), b.centroids.view(np.uint32)) for a, b in zip(both, host))
    assert both[1].centroids.size == 8 and np.all(np.diff(both[1].centroids) > 0)


def test_samples_are_there_again_for_the_passes_over_all(tq):
    """The second fit's samples take the place of the first one's; where that one then has to go over all of its own after all
    (magnitudes in one or two buckets, their residuals in many), it finds them there."""
    torch = pytest.importorskip("torch")
    rows, cols = 40_000, 64
    g = torch.Generator(device="cuda").manual_seed(11)
    w = torch.randn((rows, cols), generator=g, device="cuda") * (2e-3 / 8)
    w[:, 5] += 1.0                                          # its transform: +-1 in every column
    both = tq.fit_layer_codebooks(w, cols, 4, 4, 15)
    alone, _ = tq.fit_layer_codebooks(w, cols, 4, 0, 15)
    assert np.array_equal(both[0].centroids.view(np.uint32), alone.centroids.view(np.uint32))
    assert abs(np.abs(both[0].centroids - 1.0).min()) < 1e-2   # (the samples are what the test takes them for)


@pytest.mark.parametrize("rows,cols,log2_buckets", [(1024, 1024, 16), (4096, 4096, 20)])
def test_memory_kept_after_a_layer_fit(tq, rows, cols, log2_buckets):
    """Three arrays of samples, two sets of buckets, one of the CTAs' places (32 exponents or 48 K counters, for 8192 samples and more), in
    size classes an eighth wide."""
    torch = pytest.importorskip("torch")
    w = torch.randn((rows, cols), device="cuda") * 0.02
    n = rows * cols
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    places = min(sms, -(-n // 8192)) * 4 * min(49152, 64 << (log2_buckets - 9))
    tq.fit_layer_codebooks(w, 64, 4, 4, 2)
    tq.release_cached_memory()
    tq.fit_layer_codebooks(w, 64, 4, 4, 2)
    assert tq.release_cached_memory() <= 1.125 * (3 * 4 * n + 2 * 21 * 2 ** log2_buckets + places) + (1 << 20)


def test_a_fit_leaves_other_kept_memory_alone(tq):
    """A layer's fits of 1 M samples need 22 MB: caches of the other 486 MB that are kept stay."""
    torch = pytest.importorskip("torch")
    w = torch.randn((1024, 1024), device="cuda") * 0.02
    kv = torch.zeros((16, 2, 128), device="cuda", dtype=torch.float16)

    def caches(n):
        made = [tq.TQKVCache(1, 2, 128) for _ in range(n)]
        for c in made:
            c.reserve(0, 400_000)
            c.append(0, kv, kv)
        torch.cuda.synchronize()
        return made

    def close(made):
        for c in made:
            c.close()
        torch.cuda.synchronize()

    tq.fit_layer_codebooks(w, 128, 4, 4, 2)
    tq.release_cached_memory()
    close(caches(1))
    each = tq.release_cached_memory()
    n = (486 << 20) // each
    close(caches(n))
    tq.fit_layer_codebooks(w, 128, 4, 4, 2)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    made = caches(n)
    assert torch.cuda.mem_get_info()[0] > free - (32 << 20)
    close(made)
    tq.release_cached_memory()
