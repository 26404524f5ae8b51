"""Moments and limits where the estimates' tiles change: one CTA a tile (both moments in a launch) and
several, tiles of 4 to 64 dimensions, more counts to set than the limits' CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# (errors as in the estimates' other tests: FP64 sums of words good to 2^-60, a division and a
# subtraction, each a rounding of 2^-53 at most, and a tree of some ten FP64 additions)
@pytest.mark.parametrize("n,dim", [(1, 9), (15, 3), (17, 4), (1000, 20), (820, 5), (50, 3000), (33, 65), (4096, 256),
                                   (4099, 64), (65537, 100), (2500, 130), (100, 20001), (300, 4097)])
def test_moments_and_limits_over_the_tiles(n, dim):
    from bayadera_gb300.engine import GB300BayaderaFactory
    rng = np.random.default_rng(n + dim)
    x = (np.exp(rng.standard_normal((n, dim))) + np.arange(dim) % 7).astype(np.float32)
    v = x.astype(np.longdouble)
    mu = v.sum(axis=0) / n
    want = ((v - mu) ** 2).sum(axis=0) / n
    with GB300BayaderaFactory() as f:
        for _ in range(2):                       # the tickets are left as they were found
            mean, var = f.data_moments(x)
            assert np.all(np.abs(mean - mu) <= 16 * 2.0 ** -53 * np.abs(mu))
            assert np.all(np.abs(var - want) <= 16 * 2.0 ** -53 * want + (n == 1) * 1e-30)
            h = f.data_histogram(x, 64, 1)       # counts from 1
            assert np.array_equal(h.limits, np.stack([x.min(axis=0), x.max(axis=0)]))
            if n > 1:
                counts = h.pdf / (np.float32(64 / n) / (h.limits[1] - h.limits[0]))
                assert np.allclose(counts.sum(axis=0), n + 64, rtol=1e-4)
