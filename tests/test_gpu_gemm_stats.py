"""Per-step means of the resident GEMM form: a half-step's positions are summed by the next
launch, a chunk's last by a launch of its own; dims at the edges of the summing warps' 64, ragged
last tiles, runs shorter and longer than a captured chunk."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factory():
    from bayadera_gb300.engine import GB300BayaderaFactory
    f = GB300BayaderaFactory()
    yield f
    f.release()


@pytest.mark.parametrize("tensor", [False, True])
@pytest.mark.parametrize("D,W", [(2, 4), (2, 126), (31, 130), (37, 258), (64, 128), (65, 2050), (80, 66)])
def test_means_per_step(factory, D, W, tensor):
    from bayadera_gb300 import models as M
    rng = np.random.default_rng(D)
    B = rng.standard_normal((D, D)) / np.sqrt(D)
    P = (B @ B.T + np.eye(D)).astype(np.float32)
    sf = factory.mcmc_factory(M.mvn_precision_model(D), form="gemm", tensor=tensor)
    rows = {}
    for n in (1, 2, 3, 40, 67):
        s = sf.create_sampler(3, W, P.reshape(-1))
        s.init_position_normal(4, 0.0, 1.0)
        m = s.run_sampler(n, 2.0, return_means=True)["means"].T.astype(np.float64)
        x = s.positions().T.astype(np.float64)
        # tile sums in at most 64 fp32 additions, the rest in 64 bits, the mean rounded once
        assert np.all(np.abs(m[n - 1] - x.mean(0)) <= 65 * 2.0 ** -24 * np.abs(x).mean(0) + 1e-30)
        rows[n] = m
        s.release()
    # the same whether summed by the next launch or by a launch of its own
    for n in (1, 2, 3, 40):
        np.testing.assert_array_equal(rows[67][:n], rows[n])
    sf.release()
