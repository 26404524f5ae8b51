"""A recorded run whose per-step means do not fit under the context's memory limit leaves a sampler
and a batch whose next runs record theirs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOO_MANY = 10_000_000


def test_a_run_after_one_that_did_not_fit():
    from bayadera_gb300 import _native as N, models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    D, W = 20, 512
    P = np.eye(D, dtype=np.float32).reshape(-1)
    with GB300BayaderaFactory(mem_limit=32 << 20) as f:
        sf = f.mcmc_factory(M.mvn_precision_model(D), form="gemm")
        s = sf.create_sampler(1, W, P)
        s.init_position_normal(2, 0.0, 1.0)
        s.run_sampler(64, 2.0)                      # whole chunks: a captured graph
        with pytest.raises(N.BayaderaError):
            s.run_sampler(TOO_MANY, 2.0)
        other = sf.create_sampler(3, W, P)          # what was freed is another's now
        other.init_position_normal(4, 0.0, 1.0)
        x = other.positions()
        r = s.run_sampler(64, 2.0, return_means=True)
        assert np.allclose(r["means"][:, -1], s.positions().mean(1, dtype=np.float64), atol=1e-5)
        assert np.all(np.abs(np.diff(r["means"], axis=1)).max(axis=0) > 0.0)
        assert np.array_equal(other.positions(), x)
        for h in (other, s, sf):
            h.release()


def test_a_batch_run_after_one_that_did_not_fit():
    from bayadera_gb300 import _native as N, models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    with GB300BayaderaFactory(mem_limit=32 << 20) as f:
        sf = f.mcmc_factory(M.hierarchical_rows_batch_model(5), form="batch")
        params, rows = M.hierarchical_rows_params([np.ones(9)] * 5, np.ones(5))
        b = sf.create_batch([dict(dim=7, seed=1, walkers=256, params=params, rows=rows)])
        b.init_position_normal([2], 0.0, 1.0)
        b.run_sampler(64, 2.0)
        with pytest.raises(N.BayaderaError):
            b.run_sampler(TOO_MANY, 2.0)
        r = b.run_sampler(64, 2.0, return_means=True)
        assert np.allclose(r["means"][0][:, -1], b.positions()[0].mean(0, dtype=np.float64), atol=1e-5)
        for h in (b, sf):
            h.release()
