"""The streamed tensor-core form at the edges of its tiles: walker operand in tensor memory
(one sub-tile, up to 256 features) and in shared memory, ragged rows and walkers, the
logistic model's 16-row sums; propose and accept launches at their tile edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factory():
    from bayadera_gb300.engine import GB300BayaderaFactory
    f = GB300BayaderaFactory()
    yield f
    f.release()


def logistic_data(n, F, scale, seed):
    rng = np.random.default_rng(seed)
    X = (scale * rng.standard_normal((n, F)) / np.sqrt(F)).astype(np.float32)
    y = (rng.random(n) < 0.5).astype(np.float32)
    return X, y, np.concatenate([np.concatenate([X, y[:, None]], axis=1).reshape(-1),
                                 np.array([5.0], np.float32)])


def fp64_logistic(X, y, pos):
    eta = X.astype(np.float64) @ pos.astype(np.float64).T
    ll = y[:, None] * eta - np.maximum(eta, 0) - np.log1p(np.exp(-np.abs(eta)))
    b = pos.astype(np.float64)
    return ll.sum(0) - (b * b).sum(1) / 50.0


# |d term / d eta| <= 1 and the split products' relative error is below 2^-15, their fp32
# accumulation's 4 F 2^-24; a row's term and its part of a sum round to 2^-22 of themselves
# (eta and the softplus), the whole to a few 2^-24.
def bound(X, pos, want):
    F = X.shape[1]
    xb = np.abs(X.astype(np.float64)) @ np.abs(pos.astype(np.float64)).T
    return ((2.0 ** -15 + 4 * F * 2.0 ** -24) * xb.sum(0)
            + 2.0 ** -22 * (np.abs(X.astype(np.float64) @ pos.astype(np.float64).T) + 2.0).sum(0)
            + 2.0 ** -22 * np.abs(want) + 1e-6)


@pytest.mark.parametrize("scale", [0.5, 200.0])
@pytest.mark.parametrize("n,F,W,sub", [(1, 3, 4, 0), (15, 5, 130, 0), (16, 5, 256, 1), (17, 64, 258, 1),
                                       (127, 65, 126, 1), (129, 128, 130, 2), (1000, 129, 128, 0),
                                       (4101, 200, 300, 1), (2049, 256, 384, 0), (700, 257, 130, 0),
                                       (300, 320, 66, 1)])
def test_logistic_log_densities_at_tile_edges(factory, n, F, W, sub, scale):
    from bayadera_gb300 import models as M
    X, y, params = logistic_data(n, F, scale, n + F)
    pos = np.random.default_rng(F).standard_normal((W, F)).astype(np.float32)
    sf = factory.mcmc_factory(M.logistic_model(F), form="gemm", tensor=True, streaming=True,
                              tc_subtiles=sub)
    s = sf.create_sampler(1, W, params)
    s.init_position(pos)
    want = fp64_logistic(X, y, pos)
    assert np.all(np.abs(s.logfn() - want) <= bound(X, pos, want))
    s.release()
    sf.release()


def test_logistic_rejects_non_finite_coefficients(factory):
    from bayadera_gb300 import models as M
    X, y, params = logistic_data(200, 4, 1.0, 9)
    pos = np.random.default_rng(1).standard_normal((16, 4)).astype(np.float32)
    pos[3, 2], pos[5, 0], pos[7, 1] = np.nan, np.inf, -np.inf
    sf = factory.mcmc_factory(M.logistic_model(4), form="gemm", tensor=True, streaming=True)
    s = sf.create_sampler(1, 16, params)
    s.init_position(pos)
    bad = ~np.isfinite(s.logfn())
    assert bad[[3, 5, 7]].all() and bad.sum() == 3
    s.release()
    sf.release()


@pytest.mark.parametrize("D,W", [(9, 14), (65, 512), (66, 516), (130, 1026), (255, 40)])
def test_streamed_moves_match_the_plain_rule(factory, D, W):
    """One bare step of the streamed form: every walker is either where it was or on the line
    through its partner, its log density that of its position, as recomputed from there."""
    from bayadera_gb300 import models as M
    F = D - 1
    rng = np.random.default_rng(D)
    n = 300
    X = rng.standard_normal((n, F)).astype(np.float32)
    rows = np.concatenate([X, (X @ (rng.standard_normal(F) / F) + rng.standard_t(4, n))[:, None]], axis=1)
    params = np.concatenate([rows.reshape(-1), [4.0, 10.0, 1.0]]).astype(np.float32)
    sf = factory.mcmc_factory(M.robust_t_model(F), form="gemm", tensor=True, streaming=True)
    s = sf.create_sampler(5, W, params)
    s.init_position_normal(6, 0.0, 0.1)
    before = s.positions().T.copy()
    s.burn_in(1, 2.0)
    after, lf = s.positions().T.copy(), s.logfn()
    moved = np.any(before != after, axis=1)
    assert 0 < moved.sum() < W
    K = W // 2
    for half in (0, 1):
        own = slice(half * K, half * K + K)
        other = before[K:] if half == 0 else after[:K]
        for k in np.flatnonzero(moved[own])[:20]:
            x, y = before[own][k].astype(np.float64), after[own][k].astype(np.float64)
            # y = s + z (x - s) for one partner s and one z: (y - s) parallel to (x - s)
            u, v = y - other, x - other
            z = (u * v).sum(1) / (v * v).sum(1)
            off = np.abs(u - z[:, None] * v).max(axis=1)
            assert off.min() <= 1e-5 * (1 + np.abs(y).max())
    s.init_position(after)
    assert np.array_equal(s.logfn(), lf)
    s.release()
    sf.release()
