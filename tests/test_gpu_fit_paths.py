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
