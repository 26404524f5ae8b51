"""A histogram whose buffers do not fit under the context's memory limit leaves a sampler that can
make smaller ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_histogram_after_one_that_did_not_fit():
    from bayadera_gb300 import _native as N, models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    D, W = 200, 256
    limit, ref = 0, None
    for _ in range(2):
        with GB300BayaderaFactory(mem_limit=limit) as f:
            sf = f.mcmc_factory(M.mvn_precision_model(D), form="plain")
            s = sf.create_sampler(1, W, np.eye(D, dtype=np.float32).reshape(-1))
            s.init_position_normal(2, 0.0, 1.0)
            h = s.histogram(1, 16)
            if limit:
                with pytest.raises(N.BayaderaError):
                    s.histogram(1, 1024)             # 2.4 MB of counts and densities
                h = s.histogram(1, 16)
                assert np.array_equal(h.pdf, ref.pdf) and np.array_equal(h.limits, ref.limits)
            else:
                limit, ref = f.allocated() + (1 << 20), h
            s.release()
            sf.release()
