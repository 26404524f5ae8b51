"""The plain form's launches at the edges of their split: params staged in shared memory or
not, groups of 256 walkers as one CTA or as a cluster of four."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factory():
    from bayadera_gb300.engine import GB300BayaderaFactory
    f = GB300BayaderaFactory()
    yield f
    f.release()


def gauss_params(n):
    y = np.random.default_rng(n).normal(3.0, 2.0, n).astype(np.float32)
    return y, np.concatenate([y, np.array([0.0, 10.0, 0.0, 20.0], np.float32)])


# fp32 sum of n terms in order: n 2^-24 of their magnitudes at worst, and fast-math's few ulp
# in each term and in the log-scale.
@pytest.mark.parametrize("W", [4, 62, 130, 1026, 16388])
@pytest.mark.parametrize("n", [1, 2, 5, 16, 17, 18, 1000, 11260, 11261, 49000, 51196, 51197])
def test_log_densities_with_params_staged_or_not(factory, n, W):
    from bayadera_gb300 import models as M
    y, params = gauss_params(n)
    sf = factory.mcmc_factory(M.gaussian_posterior_model(), form="plain")
    s = sf.create_sampler(3, W, params)
    s.init_position(4, [2.0, 4.0, 1.0, 3.0])
    s.burn_in(2, 2.0)
    pos = s.positions().T.astype(np.float64)
    mu, sg = pos[:, 0], pos[:, 1]
    k = np.arange(0, W, max(1, W // 64))
    ss = ((y[None, :].astype(np.float64) - mu[k, None]) ** 2).sum(1) / (2 * sg[k] ** 2)
    c = 0.5 * np.log(2 * np.pi)
    want = -ss - n * (np.log(sg[k]) + c) - mu[k] ** 2 / 200.0 - np.log(10.0) - c - np.log(20.0)
    size = ss + n * (np.abs(np.log(sg[k])) + c) + 10.0
    assert np.all(np.abs(s.logfn()[k] - want) <= (n * 2.0 ** -24 + 2.0 ** -20) * size)
    s.release()
    sf.release()


# The split changes neither a walker's arithmetic nor the order of the statistics: a group of
# 256 walkers sums its 8 warps in order whether they are one CTA or four.  512-thread groups
# (never split) give the same walkers, and means that differ by fp32 partial sums only.
@pytest.mark.parametrize("D,W", [(1, 64), (3, 514), (64, 1024), (65, 1026), (130, 700), (20, 77000),
                                 (2, 80000)])
def test_split_groups_move_and_count_like_whole_ones(factory, D, W):
    from bayadera_gb300 import models as M
    rng = np.random.default_rng(D)
    A = rng.standard_normal((D, D)) / np.sqrt(D)
    P = (A @ A.T + np.eye(D)).astype(np.float32).reshape(-1)
    runs = []
    for cta in (0, 512):
        sf = factory.mcmc_factory(M.mvn_precision_model(D), form="plain", cta_threads=cta)
        s = sf.create_sampler(5, W, P)
        s.init_position_normal(6, 0.0, 1.0)
        s.burn_in(3, 2.0)
        r = s.run_sampler(50, 2.0, return_means=True)
        runs.append((s.positions().T.copy(), s.logfn(), r["acceptance_rate"], r["means"]))
        s.release()
        sf.release()
    (p0, l0, a0, m0), (p1, l1, a1, m1) = runs
    assert np.array_equal(p0, p1) and np.array_equal(l0, l1) and a0 == a1
    sd = p0.astype(np.float64).std()
    assert np.all(np.abs(m0 - m1) <= 2.0 ** -20 * (np.abs(m0) + sd))
    assert np.all(np.abs(m0[:, -1] - p0.astype(np.float64).mean(0)) <= 2.0 ** -20 * sd + 1e-7)
