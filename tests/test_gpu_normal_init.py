"""The normal walker init against its FP64 formula on the CPU, over means and scales that move
the rounding test's bound about (large offsets, tiny and huge scales, a zero scale)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# The CPU's FP64 log, sqrt, sin and cos and the GPU's differ by a few 2^-53, which rounds to
# another float for some 2^-27 of the values: up to 2 of the 300,000 here may be a unit off.
@pytest.mark.parametrize("mean,sd", [(0.0, 1.0), (0.0, 0.05), (3.0, 2.0), (1e4, 1.0), (-0.5, 1e-3),
                                     (0.0, 1e-22), (0.0, 1e33), (2.5, 0.0), (1e-21, 1e-21)])
@pytest.mark.parametrize("D,W", [(1, 4), (3, 50002), (7, 42858)])
def test_normal_init_is_the_fp64_formula(oracle, D, W, mean, sd):
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import GB300BayaderaFactory
    with GB300BayaderaFactory() as f:
        sf = f.mcmc_factory(M.mvn_precision_model(D), form="plain")
        s = sf.create_sampler(1, W, np.eye(D, dtype=np.float32).reshape(-1))
        s.init_position_normal(12, mean, sd)
        got = s.positions().T.copy()
        s.release()
        sf.release()
    r = oracle.Stretch("mvn_precision", D, W, np.eye(D, dtype=np.float32).reshape(-1), seed=1)
    r.init_position_normal(12, mean, sd)
    want = r.xs.reshape(W, D)
    assert (got != want).sum() <= 2
    with np.errstate(over="ignore"):
        assert np.allclose(got, want, rtol=2.0 ** -22, atol=0.0)
