"""Device memory that a context keeps between calls: what fits under its limit without the kept
memory fits with it, and a call's need is known from its first time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def series(mb):
    """Two series whose autocorrelation call stages and works on mb MiB."""
    n = mb * MB // 24
    return np.random.default_rng(mb).standard_normal((2, n)).astype(np.float32)


def points(mb):
    """mb MiB of points (mu, sigma)."""
    n = mb * MB // 8
    x = np.random.default_rng(mb).standard_normal((n, 2)).astype(np.float32)
    x[:, 1] = 1.0 + np.abs(x[:, 1])
    return x


@pytest.mark.parametrize("call", ["log_density", "evidence", "moments", "histogram"])
def test_a_call_that_fits_alone_fits_beside_the_kept_block(call):
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    x, y = points(60), np.float32([0.5, 1.5, 2.5])
    with GB300BayaderaFactory(mem_limit=98 * MB) as f:
        e = f.likelihood_engine(M.likelihood_models()["gaussian"], 2)
        for _ in range(4):
            f.acor(series(56))
        assert f.allocated() >= 55 * MB          # kept
        if call == "log_density":                # 60 MiB of points, 30 of densities
            got = e.log_density(y, x)
            want = sum(-(np.float64(v) - x[::997, 0]) ** 2 / (2.0 * x[::997, 1].astype(np.float64) ** 2)
                       - np.log(x[::997, 1]) - 0.5 * np.log(2 * np.pi) for v in y)
            assert np.allclose(got[::997], want, rtol=1e-5, atol=1e-5)
        elif call == "evidence":
            assert 0.0 < e.evidence(y, x) < 1.0
        elif call == "moments":
            assert np.allclose(f.data_moments(x)[0], x.mean(0, dtype=np.float64), atol=1e-9)
        else:
            assert np.array_equal(f.data_histogram(x, 64).limits, np.stack([x.min(0), x.max(0)]))
        assert f.allocated() <= 98 * MB
        e.release()


def test_a_call_settles_what_is_kept_the_first_time():
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    with GB300BayaderaFactory() as f:
        f.data_moments(points(1))
        held = [f.allocated()]
        for m in (series(12), series(12), series(3), series(12)):
            f.acor(m)
            held.append(f.allocated())
        # the larger need replaces the first one's block; the estimates' workspace stays
        assert held[1] >= 12 * MB - 64 and held[1] <= held[0] + 12 * MB
        assert held[1:] == [held[1]] * 4
        # nothing is kept of a call that needs more than the bound in all, its parts included
        e = f.likelihood_engine(M.likelihood_models()["gaussian"], 2)
        for _ in range(3):
            e.log_density(np.float32([0.0]), points(50))      # 75 MiB
            assert f.allocated() == held[1]
        e.release()


def test_with_its_last_handle_a_context_gives_everything_back():
    """A host's leak check: what is allocated after the handles' release is what was before."""
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    with GB300BayaderaFactory() as f:
        before = f.allocated()
        sf = f.mcmc_factory(M.mvn_precision_model(5), form="gemm")
        a, b = (sf.create_sampler(i, 512, np.eye(5, dtype=np.float32).reshape(-1)) for i in (1, 2))
        for s in (a, b):
            s.init_position_normal(3, 0.0, 1.0)
            s.run_sampler(60, 2.0)
            s.sd()
            s.histogram(1, 64)
        f.acor(series(3))
        held = f.allocated()
        a.release()
        assert 3 * MB < f.allocated() < held              # kept for the other one
        b.release()
        assert f.allocated() == before
        sf.release()
        sf = f.mcmc_factory(M.hierarchical_rows_batch_model(3), form="batch")
        params, rows = M.hierarchical_rows_params([np.ones(9)] * 3, np.ones(3))
        h = sf.create_batch([dict(dim=5, seed=1, walkers=64, params=params, rows=rows)])
        h.init_position_normal([2], 0.0, 1.0)
        h.burn_in(2, 2.0)
        f.acor(series(1))
        h.release()
        assert f.allocated() == before
        sf.release()
