"""The resident tensor-core form at the edges of its gather and its CTAs: rows taken in items of
2, 4 and 8 dims (at most 64 dims and even, or not), K steps of zeros left out, one or two tile
groups a CTA by the sampler's choice, ragged last tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factory():
    from bayadera_gb300.engine import GB300BayaderaFactory
    f = GB300BayaderaFactory()
    yield f
    f.release()


def precision(D):
    rng = np.random.default_rng(D)
    B = rng.standard_normal((D, D)) / np.sqrt(D)
    return (B @ B.T + np.eye(D)).astype(np.float32)


def run(factory, D, W, burn, **kw):
    from bayadera_gb300 import models as M
    sf = factory.mcmc_factory(M.mvn_precision_model(D), form="gemm", **kw)
    s = sf.create_sampler(3, W, precision(D).reshape(-1))
    s.init_position_normal(4, 0.0, 1.0)
    s.burn_in(burn, 2.0)
    pos, logfn = s.positions().copy(), s.logfn().copy()
    r = s.run_sampler(5, 2.0, return_means=True)
    out = (pos, logfn, r["means"].copy(), r["acceptance_rate"], s.positions().copy())
    s.release()
    sf.release()
    return out


@pytest.mark.parametrize("D,W", [(2, 130), (3, 66), (4, 128), (6, 254), (16, 1000), (17, 130), (18, 134),
                                 (48, 142), (62, 390), (63, 390), (64, 19594), (65, 19594), (66, 258),
                                 (96, 19594), (97, 19458), (98, 19594), (99, 130), (128, 19594),
                                 (128, 2 * 64 * 305 + 2)])
def test_gather_groups_and_log_densities(factory, D, W):
    pos, logfn, means, rate, last = run(factory, D, W, 2, tensor=True)
    # the same for one and for two groups a CTA
    for groups in (1, 2):
        other = run(factory, D, W, 2, tensor=True, tc_groups=groups)
        for x, y in zip((pos, logfn, means, last), (other[0], other[1], other[2], other[4])):
            np.testing.assert_array_equal(x, y)
        assert rate == other[3]
    # log densities: the split products are good to 2^-15 of each, their fp32 sum to 4 D 2^-24,
    # the row terms and their sum to 2^-21
    P, x = precision(D).astype(np.float64), pos.T.astype(np.float64)
    want = -0.5 * np.einsum("wi,ij,wj->w", x, P, x)
    terms = 0.5 * np.einsum("wi,ij,wj->w", np.abs(x), np.abs(P), np.abs(x))
    assert np.all(np.abs(logfn - want) <= (2.0 ** -15 + 4 * D * 2.0 ** -24 + 2.0 ** -21) * terms + 1e-6)
    # the moves: the fp32 form's, but for decisions within the densities' error (two steps;
    # about 2^-15 of some D a decision, far below one in a hundred)
    ref = run(factory, D, W, 2, tensor=False)[0].T
    differ = np.count_nonzero(np.any(x != ref.astype(np.float64), axis=1))
    assert differ <= max(2, W // 50), differ
