"""The estimate kernels (moments, limits, histograms) at the sizes where their split changes:
one and several dimension tiles, one and several CTAs a tile, ragged rows, and values that
leave the fp32 batches' range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factory():
    from bayadera_gb300.engine import GB300BayaderaFactory
    f = GB300BayaderaFactory()
    yield f
    f.release()


def matrix(n, dim, kind):
    rng = np.random.default_rng(1000 * dim + n)
    x = rng.standard_normal((n, dim))
    if kind == "offset":
        x = x + 1e4 * (1 + np.arange(dim))
    elif kind == "huge":
        x = x * 1e30
    elif kind == "tiny":
        x = x * 1e-30
    elif kind == "mixed":
        x[:: max(1, n // 7)] *= 1e18
    return x.astype(np.float32)


SHAPES = [(1, 1), (5, 3), (16, 256), (17, 257), (255, 1), (4095, 1), (4097, 2), (40001, 7),
          (3001, 50), (700, 300), (33, 1000), (300007, 1), (60013, 6)]


# A mean's error: FP64 additions over a tree (below 2^-49 of the mean absolute value at
# these sizes) and 2^-47 for a batch's fp32 error words; a variance's the same of itself (the
# deviations are exact): 1e-12 covers every case by a factor above 50.
@pytest.mark.parametrize("kind", ["normal", "offset", "huge", "tiny", "mixed"])
@pytest.mark.parametrize("n,dim", SHAPES)
def test_moments_match_long_double(factory, n, dim, kind):
    x = matrix(n, dim, kind)
    mean, var = factory.data_moments(x)
    v = x.astype(np.longdouble)
    mu = v.sum(axis=0) / n
    want = ((v - mu) ** 2).sum(axis=0) / n
    assert np.all(np.abs(mean - mu) <= 1e-12 * np.abs(v).mean(axis=0))
    assert np.all(np.abs(var - want) <= 1e-12 * want)


def test_moments_of_constants_and_non_finite_columns(factory):
    x = matrix(5000, 6, "normal")
    x[:, 0] = 3.7
    x[17, 1] = np.inf
    x[18, 2] = np.nan
    x[19, 3] = -np.inf
    x[20, 3] = np.inf
    x[:, 4] = 3e38
    mean, var = factory.data_moments(x)
    assert mean[0] == np.float32(3.7) and 0.0 <= var[0] < 1e-28
    assert mean[1] == np.inf and np.isnan(var[1])
    assert np.isnan(mean[2]) and np.isnan(var[2]) and np.isnan(mean[3])
    assert abs(mean[4] / np.float64(np.float32(3e38)) - 1) < 1e-14
    assert abs(var[5] / x[:, 5].astype(np.float64).var() - 1) < 1e-12


@pytest.mark.parametrize("flags", [0, 1])
@pytest.mark.parametrize("bins", [2, 64, 1024])
@pytest.mark.parametrize("n,dim", SHAPES[1:])
def test_histogram_matches_float32_binning(factory, n, dim, bins, flags):
    x = matrix(n, dim, "normal")
    h = factory.data_histogram(x, bins, flags)
    lo, hi = x.min(axis=0), x.max(axis=0)
    assert np.array_equal(h.limits, np.stack([lo, hi]))
    b = ((x - lo) / (hi - lo) * np.float32(bins)).astype(np.uint32)
    b = np.minimum(b, bins - 1)
    counts = np.stack([np.bincount(c, minlength=bins) for c in b.T], axis=1) + flags
    scale = np.float32(bins / n) / (hi - lo)
    assert np.array_equal(h.pdf, scale * counts.astype(np.float32))
    order = np.take_along_axis(h.pdf, h.bin_ranks.astype(np.int64), axis=0)
    assert np.all(np.diff(order, axis=0) <= 0)
    assert np.array_equal(np.sort(h.bin_ranks, axis=0),
                          np.repeat(np.arange(bins, dtype=np.float32)[:, None], dim, axis=1))


def test_limits_pass_over_nan(factory):
    x = matrix(3000, 3, "normal")
    x[0, 0] = np.nan
    x[2999, 1] = np.nan
    x[:, 2] = np.nan
    h = factory.data_histogram(x, 16)
    assert h.limits[0, 0] == np.nanmin(x[:, 0]) and h.limits[1, 1] == np.nanmax(x[:, 1])
    assert np.all(np.isnan(h.limits[:, 2]))


# FP64 sums of n lag terms in another order than the oracle's: n lag 2^-53 is 3e-10 at the
# longest series, and a random walk of the roundings some 1e-13.
@pytest.mark.parametrize("rho", [0.0, 0.97])
@pytest.mark.parametrize("wgs", [64, 1024])
@pytest.mark.parametrize("n", [50, 51, 127, 320, 1024, 1025, 2049, 4224, 16385, 40003])
def test_acor_matches_oracle_at_the_split_edges(oracle, n, wgs, rho):
    from bayadera_gb300.engine import GB300BayaderaFactory
    rng = np.random.default_rng(n)
    x = rng.standard_normal((3, n))
    for t in range(1, n):
        x[:, t] += rho * x[:, t - 1]
    x = x.astype(np.float32)
    with GB300BayaderaFactory(wgs=wgs) as f:
        got = f.acor(x)
    tau, mean, sigma, lag = oracle.acor64(x, wgs)
    assert got.lag == lag
    assert np.allclose(got.tau, tau, rtol=1e-11, atol=0)
    assert np.allclose(got.sigma, sigma, rtol=1e-11, atol=0, equal_nan=True)
    assert np.allclose(got.mean, mean, rtol=0, atol=1e-13 * np.abs(x).max())


# Skewed columns, whose fp32 rounding errors do not cancel: three levels of FP64 sums, a
# division and a subtraction, each a rounding of 2^-53 at most, beside words good to 2^-60.
@pytest.mark.parametrize("n", [1000, 8192, 262147, 2000003])
def test_moments_of_skewed_columns_to_fp64_rounding(factory, n):
    rng = np.random.default_rng(n)
    z = rng.standard_normal((n, 3))
    x = (np.stack([z[:, 0] ** 2, np.exp(2.0 * z[:, 1]), np.sign(z[:, 2]) * z[:, 2] ** 2 - 5.0], 1)
         * [1.0, 1.0, 1.5]).astype(np.float32)
    q = x.astype(np.longdouble)
    mean = q.mean(0)
    var = ((q - mean) ** 2).mean(0)
    got_mean, got_var = factory.data_moments(x)
    assert np.all(np.abs(got_mean - mean) <= 6 * 2.0 ** -53 * np.abs(mean))
    assert np.all(np.abs(got_var - var) <= 6 * 2.0 ** -53 * var)


def test_scratch_is_kept_bounded_and_given_back(oracle):
    """The kept call scratch: repeated calls of mixed sizes give the same results, it stays
    below its bound, and a context at its memory limit gets it back for a sampler."""
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    rng = np.random.default_rng(3)
    small = rng.standard_normal((2, 500)).astype(np.float32)
    large = rng.standard_normal((2, 4_000_000)).astype(np.float32)      # 96 MB of work
    with GB300BayaderaFactory() as f:
        first = [f.acor(m).tau for m in (small, large, small)]
        for _ in range(2):
            for m, t in zip((small, large, small), first):
                assert np.array_equal(f.acor(m).tau, t)
                assert np.array_equal(f.acor(np.asfortranarray(m)).tau, t)
        assert f.allocated() <= (64 << 20) + (3 << 20)
    limit = 24 << 20
    with GB300BayaderaFactory(mem_limit=limit) as f:
        mid = rng.standard_normal((2, 500_000)).astype(np.float32)      # 4 MB + 8 MB
        for _ in range(3):
            f.acor(mid)
        assert f.allocated() > 8 << 20
        sf = f.mcmc_factory(M.mvn_precision_model(40), form="plain")
        s = sf.create_sampler(1, 131072, np.eye(40, dtype=np.float32).reshape(-1))   # 21 MB
        assert f.allocated() <= limit
        s.release()
        sf.release()
