"""Plain-form model sources that are not plain C all through: what they did before the params were
staged in shared memory they do still."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# -sum (x - d_i)^2 over the data, by way of a table in shared memory of the source's own
SHARED = """
extern "C" {
inline REAL with_table(const uint32_t data_len, const uint32_t params_len, const REAL* params,
                       const uint32_t dim, const REAL* x) {
    __shared__ REAL table[10000];
    table[threadIdx.x] = x[0];
    REAL acc = 0.0f;
    for (uint32_t i = 0; i < data_len; ++i) {
        const REAL d = table[threadIdx.x] - params[i];
        acc -= d * d;
    }
    return acc;
}
}
"""


def run(f, source, logfn, data, W=64, steps=4):
    from bayadera_gb300 import models as M
    m = M.device_distribution_model(source, name=logfn, logpdf=logfn, dimension=1, params_size=0)
    sf = f.mcmc_factory(m, form="plain")
    s = sf.create_sampler(3, W, data)
    s.init_position(4, [-1.0, 1.0])
    s.burn_in(steps, 2.0)
    s.run_sampler(50, 2.0)
    x, lf = s.positions()[0].astype(np.float64), s.logfn()
    e = f.distribution_engine(m)
    points = np.linspace(-2.0, 2.0, 1000, dtype=np.float32)[:, None]
    ld = e.log_density(data, points)
    for h in (e, s, sf):
        h.release()
    return x, lf, points[:, 0].astype(np.float64), ld


def check(got, data):
    x, lf, p, ld = got
    d = data.astype(np.float64)[:, None]
    # fp32 sums of n squares, and the squares' own roundings
    for v, g in ((x, lf), (p, ld)):
        want = -((v - d) ** 2).sum(0)
        assert np.all(np.abs(g - want) <= (len(data) + 4) * 2.0 ** -24 * np.abs(want))


def test_a_source_with_shared_memory_of_its_own():
    from bayadera_gb300.engine import GB300BayaderaFactory
    data = np.random.default_rng(1).standard_normal(100).astype(np.float32)
    with GB300BayaderaFactory() as f:
        check(run(f, SHARED, "with_table", data), data)
