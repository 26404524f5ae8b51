"""A source that is given global rows and params walks as the same source given shared ones does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PASTE = "#define UNUSED_PASTE(a, b) a##b\n"    # such a source is given global memory


@pytest.fixture(scope="module")
def factory():
    from bayadera_gb300.engine import GB300BayaderaFactory
    f = GB300BayaderaFactory()
    yield f
    f.release()


def pair(model):
    yield model
    model.sources = [PASTE] + model.sources
    yield model


@pytest.mark.parametrize("D,W", [(7, 14), (65, 514), (1500, 10), (1600, 6)])
def test_streamed_moves(factory, D, W):
    from bayadera_gb300 import models as M
    rng = np.random.default_rng(D)
    P = (np.eye(D) + 0.1 / D).astype(np.float32)
    F = min(D, 8)
    gemm = dict(M.mvn_precision_model(F).gemm)
    out = []
    for m in pair(M.device_distribution_model(M.get_source("mvn_precision"), name="mvn", dimension=D, params_size=F * F,
                                              logpdf="mvn_precision_logpdf", gemm=gemm)):
        sf = factory.mcmc_factory(m, form="gemm", streaming=True)
        s = sf.create_sampler(3, W, np.ascontiguousarray(P[:F, :F]).reshape(-1))
        s.init_position_normal(4, 0.0, 1.0)
        s.burn_in(3, 2.0)
        s.run_sampler(50, 2.0)
        out.append((s.positions(), s.logfn()))
        s.release()
        sf.release()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("wpt", [1, 4])
def test_batch_moves(factory, wpt):
    from bayadera_gb300 import models as M
    rng = np.random.default_rng(wpt)
    members = []
    for i, (J, W) in enumerate([(2, 4), (5, 66), (40, 130)]):
        ys = [rng.normal(0.0, 1.0, rng.integers(5, 60)) for _ in range(J)]
        params, rows = M.hierarchical_rows_params(ys, np.ones(J))
        members.append(dict(dim=J + 2, seed=i, walkers=W, params=params, rows=rows))
    out = []
    for m in pair(M.hierarchical_rows_batch_model(40)):
        sf = factory.mcmc_factory(m, form="batch")
        b = sf.create_batch(members, dict(rows_per_thread=64, walkers_per_item=32, chunk_floats=4096,
                                          walkers_per_thread=wpt))
        b.init_position_normal([5, 6, 7], 0.0, 1.0)
        b.burn_in(4, 2.0)
        out.append([np.concatenate([v.reshape(-1) for v in part]) for part in (b.positions(), b.logfn())])
        b.release()
        sf.release()
    assert all(np.array_equal(u, v) for u, v in zip(*out))


@pytest.mark.parametrize("n", [3, 1000])
def test_plain_moves(factory, n):
    from bayadera_gb300 import models as M
    y = np.random.default_rng(n).normal(3.0, 2.0, n).astype(np.float32)
    out = []
    for m in pair(M.gaussian_posterior_model()):
        sf = factory.mcmc_factory(m, form="plain")
        s = sf.create_sampler(3, 516, np.concatenate([y, np.array([0.0, 10.0, 0.0, 20.0], np.float32)]))
        s.init_position(4, [2.0, 4.0, 1.0, 3.0])
        s.burn_in(5, 2.0)
        out.append((s.positions(), s.logfn()))
        s.release()
        sf.release()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
