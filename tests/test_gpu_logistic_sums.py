"""The streamed tensor-core logistic sums where the linear predictors themselves are exact: every
feature and coefficient is a bf16 value and every predictor a short one, so that the split
products and their accumulation round nothing and what is left is the row terms' own error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def log_densities(X, y, pos, sub):
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    F = X.shape[1]
    params = np.concatenate([np.concatenate([X, y[:, None]], axis=1).reshape(-1), [1e18]]).astype(np.float32)
    with GB300BayaderaFactory() as f:
        sf = f.mcmc_factory(M.logistic_model(F), form="gemm", tensor=True, streaming=True, tc_subtiles=sub)
        s = sf.create_sampler(1, len(pos), params)
        s.init_position(pos.astype(np.float32))
        got = s.logfn()
        s.release()
        sf.release()
    return got.astype(np.float64)


# Well separated data, 2 % of the labels flipped.  With y of 0 or 1 a row's y eta - max(eta, 0) is
# exactly 0 or -|eta|, and log(1 + exp(-|eta|)) < 5e-18 at |eta| >= 40.  So the sum is that of the
# flipped rows' -|eta|: 16 of them are added up with 15 roundings of 2^-24 of their magnitudes at
# most, batches by a compensated sum, and the result is a float (2^-24): 2^-20 of the sum of the
# magnitudes in all.  Rows past the last 16 take a softplus each, log(1 + 0) = 0 there.
@pytest.mark.parametrize("sub", [1, 2])
@pytest.mark.parametrize("n", [16, 1000, 20011])
def test_flipped_labels_among_well_separated_rows(n, sub):
    rng = np.random.default_rng(n)
    F, W = 3, 130
    # one feature a row: large predictors beside small ones in every batch of rows
    size = np.where(rng.random(n) < 0.5, rng.integers(40, 64, n), rng.integers(40, 64, n) * 2.0 ** 12)
    X = np.zeros((n, F))
    X[np.arange(n), rng.integers(0, F, n)] = size * rng.choice([-1.0, 1.0], n)
    pos = 1.0 + rng.integers(0, 128, (W, F)) / 128.0               # in [1, 2): the predictors' signs are X's
    flipped = (rng.random(n) < 0.02) & (size < 64)
    flipped[np.flatnonzero(size < 64)[:1]] = True
    y = (X.sum(1) > 0) ^ flipped
    want = -np.abs(X[flipped] @ pos.T).sum(0)
    got = log_densities(X, y.astype(np.float64), pos, sub)
    assert np.all(np.abs(got - want) <= 2.0 ** -20 * np.abs(want))


# The fast exponential's mean error is taken out by a constant, which a compiler may make wrong.
# The walkers' rounding errors, 2^-24 of each sum at most, average out over 1,024 of them (below
# 2^-29); what the sums are off by on average is to stay below a quarter of a float's rounding.
@pytest.mark.parametrize("n,spread", [(32768, 1.0), (32768, 0.25), (4096, 4.0)])
def test_sums_have_no_mean_error(n, spread):
    rng = np.random.default_rng(n + int(4 * spread))
    F, W = 8, 1024
    X = rng.integers(-24, 25, (n, F)) / 16.0
    pos = spread * rng.integers(-16, 17, (W, F)) / 16.0
    y = (rng.random(n) < 0.5).astype(np.float64)
    eta = X @ pos.T
    want = (y[:, None] * eta - np.logaddexp(0.0, eta)).sum(0)
    got = log_densities(X, y, pos, 1)
    assert abs(np.mean((got - want) / want)) <= 2.0 ** -26
