"""A row term's form for several rows goes with that term alone: a model whose source also
holds the built-in logistic term, but names a term of its own, gets its own, and
one with more values a row than that form reads takes the term row by row."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OWN = """
extern "C" {
inline REAL half_logistic_term(const REAL eta, const REAL* aux, const uint64_t row, const REAL* beta,
                               const REAL* prep) {
    return 0.5f * logistic_term(eta, aux, row, beta, prep);
}
}
"""


# |d term / d eta| <= 1/2 and the split products' relative error is below 2^-15, their fp32
# accumulation's 4 F 2^-24; a row's term and its part of a sum round to 2^-22 of themselves,
# the whole to a few 2^-24.
@pytest.mark.parametrize("n,F,sub", [(5, 3, 0), (16, 5, 1), (1000, 64, 2), (4101, 70, 1)])
def test_a_source_with_the_logistic_term_and_a_term_of_its_own(n, F, sub):
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    rng = np.random.default_rng(n)
    X = (rng.standard_normal((n, F)) / np.sqrt(F)).astype(np.float32)
    y = (rng.random(n) < 0.5).astype(np.float32)
    params = np.concatenate([np.concatenate([X, y[:, None]], axis=1).reshape(-1), np.array([5.0], np.float32)])
    pos = rng.standard_normal((130, F)).astype(np.float32)
    base = M.logistic_model(F)
    model = M.device_distribution_model([M.get_source("logistic"), OWN], name="half_logistic", dimension=F,
                                        params_size=1, logpdf="logistic_logpdf",
                                        gemm=dict(base.gemm, term="half_logistic_term"))
    with GB300BayaderaFactory() as f:
        sf = f.mcmc_factory(model, form="gemm", tensor=True, streaming=True, tc_subtiles=sub)
        s = sf.create_sampler(1, 130, params)
        s.init_position(pos)
        got = s.logfn()
        s.release()
        sf.release()
    X, b = X.astype(np.float64), pos.astype(np.float64)
    eta = X @ b.T
    want = 0.5 * (y[:, None] * eta - np.logaddexp(0.0, eta)).sum(0) - (b * b).sum(1) / 50.0
    bound = (0.5 * (2.0 ** -15 + 4 * F * 2.0 ** -24) * (np.abs(X) @ np.abs(b).T).sum(0)
             + 2.0 ** -22 * (np.abs(eta) + 2.0).sum(0) + 2.0 ** -22 * np.abs(want) + 1e-6)
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("aux", [0, 1, 2, 3])
def test_the_logistic_term_with_other_values_beside_the_response(aux):
    """aux values a row from the response on (none: the term reads a zero)."""
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    n, F = 1000, 6
    rng = np.random.default_rng(aux)
    X = (rng.standard_normal((n, F)) / np.sqrt(F)).astype(np.float32)
    y = (rng.random(n) < 0.5).astype(np.float32)
    rest = rng.standard_normal((n, 3)).astype(np.float32)
    params = np.concatenate([np.concatenate([X, y[:, None], rest], axis=1).reshape(-1), np.array([5.0], np.float32)])
    pos = rng.standard_normal((130, F)).astype(np.float32)
    gemm = dict(M.logistic_model(F).gemm, ld=F + 4, aux_len=aux)
    model = M.device_distribution_model(M.get_source("logistic"), name="logistic", dimension=F, params_size=1,
                                        logpdf="logistic_logpdf", gemm=gemm)
    with GB300BayaderaFactory() as f:
        sf = f.mcmc_factory(model, form="gemm", tensor=True, streaming=True)
        s = sf.create_sampler(1, 130, params)
        s.init_position(pos)
        got = s.logfn()
        s.release()
        sf.release()
    X, b = X.astype(np.float64), pos.astype(np.float64)
    eta = X @ b.T
    want = ((y[:, None] if aux else 0.0) * eta - np.logaddexp(0.0, eta)).sum(0) - (b * b).sum(1) / 50.0
    bound = ((2.0 ** -15 + 4 * F * 2.0 ** -24) * (np.abs(X) @ np.abs(b).T).sum(0)
             + 2.0 ** -22 * (np.abs(eta) + 2.0).sum(0) + 2.0 ** -22 * np.abs(want) + 1e-6)
    assert np.all(np.abs(got - want) <= bound)
