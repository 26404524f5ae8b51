"""anneal!'s launches, which carry their beta, in every form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factory():
    from bayadera_gb300.engine import GB300BayaderaFactory
    f = GB300BayaderaFactory()
    yield f
    f.release()


@pytest.mark.parametrize("form", ["plain", "tiled", "slices", "simt", "streamed", "tensor", "tensor_streamed",
                                  "tensor_persistent"])
def test_anneal_in_one_call_is_its_steps(factory, form):
    """anneal! with a schedule of 37 temperatures (a whole chunk of steps and a partial one)
    against 37 calls of one temperature each: the same state, and a burn-in after it."""
    from bayadera_gb300 import models as M
    rng = np.random.default_rng(2)
    if form in ("plain", "tiled", "slices"):
        params = np.concatenate([rng.normal(3.0, 2.0, 300), [0.0, 10.0, 0.0, 20.0]]).astype(np.float32)
        model, kw = M.gaussian_posterior_model(), {"form": "plain" if form == "plain" else "tiled",
                                                   "tile_slices": 3 if form == "slices" else 0}
    else:
        A = rng.standard_normal((12, 12))
        params = (A @ A.T / 12 + np.eye(12)).astype(np.float32).reshape(-1)
        model, kw = M.mvn_precision_model(12), {"form": "gemm", "tensor": form.startswith("tensor"),
                                                "streaming": form.endswith("streamed")}
    temps = np.linspace(40.0, 1.5, 37)
    out = []
    for whole in (True, False):
        sf = factory.mcmc_factory(model, **kw)
        s = sf.create_sampler(8, 514, params)
        s.set_persistent(form.endswith("persistent"))
        if model.dimension == 2:
            s.init_position(9, [2.0, 4.0, 1.0, 3.0])
        else:
            s.init_position_normal(9, 0.0, 1.0)
        if whole:
            s.anneal(lambda i: temps[i], 37, 2.0)
        else:
            for t in temps:
                s.anneal(lambda i: t, 1, 2.0)
        state = [v.copy() for v in s.export_state()]
        s.burn_in(2, 2.0)
        out.append(state + [v.copy() for v in s.export_state()])
        s.release()
        sf.release()
    for x, y in zip(*out):
        assert np.array_equal(x, y)
