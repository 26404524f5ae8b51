"""The work that a user of this framework has it do, as cases to be timed and compared.

Every case is one whole use of public entry points: sampler jobs in each kernel form (data
tiled, resident GEMM on the CUDA cores and on the tensor cores, streamed GEMM on the tensor
cores, batched, plain), the adaptation driver, the dataset engine, the density and evidence
engines and the autocorrelation engine.  Models, sizes, seeds and distributions are those of
bench.py, tests/ and the built-in library, or are generic.
"""
import math

import numpy as np
import torch

from bayadera_gb300 import _native as N
from bayadera_gb300 import mcmc
from bayadera_gb300 import models as M
from bayadera_gb300.engine import GB300BayaderaFactory

LOG_SQRT_2PI = 0.5 * math.log(2.0 * math.pi)
_factory = []


def factory():
    """The process's one context, as a program holds it (with_bayadera)."""
    if not _factory:
        _factory.append(GB300BayaderaFactory())
    return _factory[0]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a first look at a small data set: a few hundred walkers, a handful of steps, the
        # walkers read back; bound by launches and the latency of one call
        dict(name="gauss2d_small", kind="gauss2d", form="tiled", walkers=512, rows=500, burn=16,
             run=0, wpc=0, cta=0, slices=0, bins=0),
        # the usual whole job on a data-heavy low-dimensional posterior: burn-in, recorded run
        # with autocorrelation, estimates, histograms (bench.py's 2-D posterior)
        dict(name="gauss2d_job", kind="gauss2d", form="tiled", walkers=4096, rows=10000, burn=64,
             run=320, wpc=8, cta=128, slices=1, bins=256),
        # the same model as a user's own C source in the reference's form (one thread a
        # walker), fewer rows
        dict(name="plain_job", kind="gauss2d", form="plain", walkers=16384, rows=1000, burn=32,
             run=64, wpc=0, cta=0, slices=0, bins=256),
        # bench.py's 50-D correlated Gaussian at its full width: burn-in, recorded run, moments,
        # histograms, the walkers into a device buffer
        dict(name="mvn50_job", kind="mvn", tensor=True, dim=50, walkers=65536, burn=64, run=128,
             bins=128),
        # the same target in full fp32 (the GEMM form's default, no tensor cores), odd sizes
        dict(name="mvn37_fp32", kind="mvn", tensor=False, dim=37, walkers=12290, burn=48, run=64,
             bins=256),
        # mixing a medium target: annealing, adaptation of a, burn-in (the mix! driver)
        dict(name="mvn20_mix", kind="mix", dim=20, walkers=4096, step=16),
        # log posteriors of a whole ensemble under a large logistic regression: where a chain
        # is started from given positions, and what each of its half-steps evaluates
        dict(name="logistic_logp", kind="logistic", rows=(1 << 20) + 77, features=64,
             walkers=8192),
        # steps of a wide robust regression, matrix streamed through the tensor cores
        dict(name="robust_steps", kind="robust", rows=(1 << 19) + 301, features=256,
             walkers=4096, burn=1),
        # many hierarchical models advanced together (bench.py's family, the shape its tuner
        # picks), means and final states read back
        dict(name="hier_batch", kind="batch", members=48, burn=16, run=32, most=4096, rpt=512,
             wpi=64, chunk=8192, wpt=4),
        # moments and histograms of a large data matrix that already lies on the device
        dict(name="data_estimates", kind="data", n=(1 << 22) + 11, dim=6, bins=256),
        # log densities and evidence of a likelihood at a large prior sample
        dict(name="evidence", kind="density", n=1 << 20, rows=32),
        # autocorrelation of several long recorded series
        dict(name="acor_long", kind="acor", dim=8, n=200003, rho=0.9),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(n, lo=4):
    return max(lo, n + n % 2)


def draw(rng):
    kind = rng.choice(["tiled", "plain", "mvn", "mvn", "fp32", "mix", "logistic", "robust", "batch",
                       "data", "density", "acor"])
    if kind in ("tiled", "plain"):
        w = _even(_log(rng, 64, 16384 if kind == "plain" else 8192))
        most = 2e7 if kind == "plain" else 4e7
        rows = _log(rng, 100, min(200000, most / w))
        wpc, cta = rng.choice([(0, 0), (8, 128), (4, 256), (16, 256), (1, 64)]) if kind == "tiled" else (0, 0)
        return dict(kind="gauss2d", form=kind, walkers=w, rows=rows, burn=rng.randint(1, 64),
                    run=rng.choice([0, rng.randint(50, 128)]), wpc=wpc, cta=cta,
                    slices=rng.choice([0, 0, 2, 4]) if kind == "tiled" else 0,
                    bins=rng.choice([16, 128, 256, 1024]))
    if kind in ("mvn", "fp32"):
        tensor = kind == "mvn"
        return dict(kind="mvn", tensor=tensor, dim=rng.randint(2, 100 if tensor else 80),
                    walkers=_even(_log(rng, 128, 65536 if tensor else 16384)),
                    burn=rng.randint(1, 64), run=rng.randint(50, 128),
                    bins=rng.choice([64, 128, 256, 1024]))
    if kind == "mix":
        return dict(kind="mix", dim=rng.randint(2, 40), walkers=_even(_log(rng, 256, 8192)),
                    step=rng.randint(8, 24))
    if kind == "logistic":
        f = rng.choice([rng.randint(3, 64), rng.randint(65, 200)])
        w = _even(_log(rng, 256, 8192))
        return dict(kind="logistic", rows=_log(rng, 2000, min(1 << 20, 5.5e11 / (f * w))), features=f,
                    walkers=w)
    if kind == "robust":
        f = rng.randint(8, 256)
        w = _even(_log(rng, 256, 4096))
        return dict(kind="robust", rows=_log(rng, 20000, min(1 << 20, 5.4e11 / (f * w))), features=f,
                    walkers=w, burn=1)
    if kind == "batch":
        return dict(kind="batch", members=_log(rng, 2, 48), burn=rng.randint(4, 16),
                    run=rng.randint(4, 32), most=rng.choice([256, 1024, 4096]),
                    **rng.choice([dict(rpt=512, wpi=64, chunk=8192, wpt=4),
                                  dict(rpt=128, wpi=64, chunk=4096, wpt=1),
                                  dict(rpt=256, wpi=32, chunk=4096, wpt=4)]))
    if kind == "data":
        d = _log(rng, 1, 64)
        return dict(kind="data", n=_log(rng, 1000, (1 << 24) // d), dim=d,
                    bins=rng.choice([16, 64, 256, 1024]))
    if kind == "density":
        return dict(kind="density", n=_log(rng, 1000, 1 << 20), rows=_log(rng, 4, 32))
    d = _log(rng, 1, 16)
    return dict(kind="acor", dim=d, n=_log(rng, 1000, 1600000 // d), rho=rng.uniform(0.0, 0.97))


# ------------------------------------------------------------------ inputs
class State:
    """A case's inputs and handles; the handles go back when the program drops it."""

    def __init__(self, case, seed):
        self.case = case
        self.seed = seed
        self.handles = []

    def own(self, h):
        self.handles.append(h)
        return h

    def __del__(self):
        while self.handles:
            self.handles.pop().release()


def _gauss2d_params(case, seed):
    rng = np.random.default_rng(seed)
    y = rng.normal(3.0, 2.0, case["rows"]).astype(np.float32)
    return np.concatenate([y, np.array([0.0, 10.0, 0.0, 20.0], np.float32)])


def precision_matrix(dim, seed):
    """Sigma_ij = s_i s_j rho^|i-j|, rho = 0.9, s_i log-uniform in [0.1, 10]; its inverse."""
    rng = np.random.default_rng(seed)
    s = np.exp(rng.uniform(np.log(0.1), np.log(10.0), dim))
    i = np.arange(dim)
    return np.linalg.inv(np.outer(s, s) * 0.9 ** np.abs(i[:, None] - i[None, :])).astype(np.float32)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _logistic_inputs(case, seed):
    n, f, w, g = case["rows"], case["features"], case["walkers"], _gen(seed)
    params = torch.empty(n * (f + 1) + 1, device="cuda")
    rows = params[:n * (f + 1)].view(n, f + 1)
    rows.normal_(generator=g)
    beta = torch.randn(f, device="cuda", generator=g) / 8.0
    eta = rows[:, :f] @ beta
    rows[:, f] = (torch.rand(n, device="cuda", generator=g) < torch.sigmoid(eta)).float()
    params[-1] = 5.0
    pos = torch.randn(w, f, device="cuda", generator=g) * 0.05
    return params, pos


def _robust_inputs(case, seed):
    n, f, g = case["rows"], case["features"], _gen(seed)
    params = torch.empty(n * (f + 1) + 3, device="cuda")
    rows = params[:n * (f + 1)].view(n, f + 1)
    scale = torch.exp((torch.rand(f, device="cuda", generator=g) * 2.0 - 1.0) * math.log(100.0))
    beta = torch.randn(f, device="cuda", generator=g) / (scale * 16.0)
    rows.normal_(generator=g)
    rows[:, :f] *= scale
    z = torch.randn(n, 5, device="cuda", generator=g)
    t4 = z[:, 0] / torch.sqrt((z[:, 1:] ** 2).sum(dim=1) / 4.0)
    rows[:, f] = rows[:, :f] @ beta + 0.5 * t4
    params[-3:] = torch.tensor([4.0, 10.0, 1.0], device="cuda")
    return params


def _batch_members(case, seed):
    """bench.py's hierarchical family: J log-uniform in [2, 128] groups, n_j log-uniform in
    [10, 1000] observations each, known sigma_j; the sizes depend on the case alone."""
    size, rng = np.random.default_rng(case["members"]), np.random.default_rng(seed)
    out = []
    for m in range(case["members"]):
        J = int(round(np.exp(size.uniform(np.log(2.0), np.log(128.0)))))
        nj = np.round(np.exp(size.uniform(np.log(10.0), np.log(1000.0), J))).astype(int)
        sig = np.exp(rng.uniform(np.log(0.5), np.log(2.0), J))
        theta = rng.normal(rng.normal(0.0, 3.0), np.exp(rng.normal(0.0, 0.5)), J)
        ys = [rng.normal(theta[j], sig[j], nj[j]) for j in range(J)]
        params, rows = M.hierarchical_rows_params(ys, sig)
        walkers = int(size.choice([w for w in (256, 512, 1024, 4096) if w <= case["most"]]))
        out.append(dict(dim=J + 2, seed=1000 + m, walkers=walkers, params=params, rows=rows))
    return out


def _data_matrix(case, seed):
    """Columns of different centre, scale and shape, one of them heavy-tailed."""
    g = _gen(seed)
    x = torch.randn(case["n"], case["dim"], device="cuda", generator=g)
    k = torch.arange(case["dim"], device="cuda", dtype=torch.float32)
    x[:, 0] = torch.sign(x[:, 0]) * x[:, 0] ** 2
    return x * (1.0 + 0.5 * k) + (10.0 * k - 5.0)


def _density_inputs(case, seed):
    rng = np.random.default_rng(seed)
    y = rng.normal(1.0, 1.0, case["rows"]).astype(np.float32)
    x = np.empty((case["n"], 2), np.float32)   # (mu, sigma) from a prior
    x[:, 0] = rng.normal(0.0, 2.0, case["n"])
    x[:, 1] = rng.uniform(0.5, 5.0, case["n"])
    return y, x


def _acor_series(case, seed):
    rng = np.random.default_rng(seed)
    e = rng.standard_normal((case["dim"], case["n"] + 256)).astype(np.float32)
    k = case["rho"] ** np.arange(256)
    return np.stack([np.convolve(r.astype(np.float64), k, "valid")[:case["n"]]
                     for r in e]).astype(np.float32)


def prepare(case, seed):
    s = State(case, seed)
    f = factory()
    kind = case["kind"]
    if kind == "gauss2d":
        s.params = _gauss2d_params(case, seed)
        sf = s.own(f.mcmc_factory(M.gaussian_posterior_model(), form=case["form"],
                                  walkers_per_cta=case["wpc"], cta_threads=case["cta"],
                                  tile_slices=case["slices"]))
        s.sampler = s.own(sf.create_sampler(seed, case["walkers"], s.params))
    elif kind in ("mvn", "mix"):
        P = precision_matrix(case["dim"], seed)
        sf = s.own(f.mcmc_factory(M.mvn_precision_model(case["dim"]), form="gemm",
                                  tensor=case.get("tensor", True)))
        s.sampler = s.own(sf.create_sampler(seed, case["walkers"], P.reshape(-1)))
        s.out = torch.empty(case["walkers"], case["dim"], device="cuda")
    elif kind == "logistic":
        params, pos = _logistic_inputs(case, seed)
        torch.cuda.synchronize()
        sf = s.own(f.mcmc_factory(M.logistic_model(case["features"]), form="gemm", tensor=True))
        s.sampler = s.own(sf.create_sampler(seed, case["walkers"], params))
        s.positions = pos.cpu().numpy()
    elif kind == "robust":
        params = _robust_inputs(case, seed)
        torch.cuda.synchronize()
        sf = s.own(f.mcmc_factory(M.robust_t_model(case["features"]), form="gemm", tensor=True))
        s.sampler = s.own(sf.create_sampler(seed, case["walkers"], params))
        s.out = torch.empty(case["walkers"], case["features"] + 1, device="cuda")
    elif kind == "batch":
        members = _batch_members(case, seed)
        sf = s.own(f.mcmc_factory(M.hierarchical_rows_batch_model(128), form="batch"))
        s.batch = s.own(sf.create_batch(members, dict(rows_per_thread=case["rpt"],
                                                      walkers_per_item=case["wpi"],
                                                      chunk_floats=case["chunk"],
                                                      walkers_per_thread=case["wpt"])))
        s.seeds = [seed + 7 + i for i in range(len(members))]
    elif kind == "data":
        s.x = _data_matrix(case, seed)
        torch.cuda.synchronize()
        d, b = case["dim"], case["bins"]
        s.mean, s.var = np.zeros(d), np.zeros(d)
        s.limits = np.zeros((d, 2), np.float32)
        s.pdf, s.ranks = np.zeros((d, b), np.float32), np.zeros((d, b), np.float32)
    elif kind == "density":
        s.y, s.x = _density_inputs(case, seed)
        s.engine = s.own(f.likelihood_engine(M.likelihood_models()["gaussian"], 2))
    else:
        s.series = _acor_series(case, seed)
    return s


# ------------------------------------------------------------------ one pass
def _job(s, init):
    """init!, walkers, burn-in, recorded run, moments, histograms."""
    c, smp = s.case, s.sampler
    smp.init(s.seed)
    init(smp)
    smp.burn_in(c["burn"], 2.0)
    out = {}
    if c["run"]:
        r = smp.run_sampler(c["run"], 2.0, return_means=True)
        ac = r["autocorrelation"]
        h = smp.histogram(1, c["bins"])
        out = dict(rate=r["acceptance_rate"], means=r["means"], tau=ac.tau, acor_mean=ac.mean,
                   sigma=ac.sigma, mean=smp.mean(), sd=smp.sd(), limits=h.limits, pdf=h.pdf,
                   ranks=h.bin_ranks)
    return out


def run(s):
    c = s.case
    kind = c["kind"]
    if kind == "gauss2d":
        out = _job(s, lambda smp: smp.init_position(s.seed + 1, [2.0, 4.0, 1.0, 3.0]))
        out["positions"] = s.sampler.positions()
        out["logfn"] = s.sampler.logfn()
        return out
    if kind == "mvn":
        out = _job(s, lambda smp: smp.init_position_normal(s.seed + 1, 0.0, 1.0))
        out["sample"] = s.sampler.sample_into(s.out)
        out["logfn"] = s.sampler.logfn()
        return out
    if kind == "mix":
        s.sampler.init(s.seed)
        s.sampler.init_position_normal(s.seed + 1, 0.0, 1.0)
        r = mcmc.mix(s.sampler, {"step": c["step"]})
        return dict(r, sample=s.sampler.sample_into(s.out), logfn=s.sampler.logfn())
    if kind == "logistic":
        s.sampler.init_position(s.positions)
        return s.sampler.logfn()
    if kind == "robust":
        s.sampler.init(s.seed)
        s.sampler.init_position_normal(s.seed + 1, 0.0, 0.01)
        s.sampler.burn_in(c["burn"], 2.0)
        return dict(sample=s.sampler.sample_into(s.out), logfn=s.sampler.logfn())
    if kind == "batch":
        s.batch.init_position_normal(s.seeds, 0.0, 1.0)
        s.batch.burn_in(c["burn"], 2.0)
        r = s.batch.run_sampler(c["run"], 2.0, return_means=True)
        return dict(rates=r["acceptance_rates"],
                    means=np.concatenate([m.T.reshape(-1) for m in r["means"]]),
                    positions=np.concatenate([p.reshape(-1) for p in s.batch.positions()]),
                    logfn=np.concatenate(s.batch.logfn()))
    if kind == "data":
        # the C ABI takes data on the device, as a JVM host passes it
        ctx, n, d = factory().ctx, c["n"], c["dim"]
        p = N.C.c_void_p
        N.call("bay_data_moments", ctx, p(s.x.data_ptr()), d, n, p(s.mean.ctypes.data),
               p(s.var.ctypes.data))
        N.call("bay_data_histogram", ctx, p(s.x.data_ptr()), d, n, c["bins"], 0,
               p(s.limits.ctypes.data), p(s.pdf.ctypes.data), p(s.ranks.ctypes.data))
        return dict(mean=s.mean, variance=s.var, limits=s.limits, pdf=s.pdf, ranks=s.ranks)
    if kind == "density":
        return dict(log_density=s.engine.log_density(s.y, s.x), evidence=s.engine.evidence(s.y, s.x))
    r = factory().acor(s.series)
    return dict(tau=r.tau, mean=r.mean, sigma=r.sigma)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c, kind = case, case["kind"]
    if kind == "gauss2d":
        w, steps = c["walkers"], c["burn"] + c["run"] + 1
        return {"bytes": 4.0 * c["rows"] + 24.0 * w, "flops": 3.0 * c["rows"] * w * steps}
    if kind in ("mvn", "mix"):
        d, w = c["dim"], c["walkers"]
        if kind == "mvn":
            steps = c["burn"] + c["run"] + 2
        else:
            steps = 2 * int(c["step"] * d ** 0.8) + c["step"] + 6
        return {"bytes": (12.0 * d + 8.0) * w * steps, "flops": 2.0 * d * d * w * steps}
    if kind in ("logistic", "robust"):
        n, f, w = c["rows"], c["features"], c["walkers"]
        evals = 1 if kind == "logistic" else c["burn"] + 2
        return {"bytes": 4.0 * n * (f + 1) * evals + 4.0 * w * f, "flops": 2.0 * n * f * w * evals}
    if kind == "batch":
        mem = _batch_members(c, 0)
        steps = c["burn"] + c["run"] + 1
        fl = sum(m["walkers"] * 3.0 * (m["rows"] + m["dim"]) for m in mem)
        return {"bytes": sum(8.0 * m["walkers"] * m["dim"] + 4.0 * m["params"].size for m in mem),
                "flops": fl * steps}
    if kind == "data":
        return {"bytes": 4.0 * c["n"] * c["dim"], "flops": 12.0 * c["n"] * c["dim"]}
    if kind == "density":
        return {"bytes": 12.0 * c["n"], "flops": 2.0 * 3.0 * c["n"] * c["rows"]}
    return {"bytes": 4.0 * c["dim"] * c["n"], "flops": 8.0 * c["dim"] * c["n"]}


# ------------------------------------------------------------------ the same in 64 bits
def _acor64(series, wgs=1024):
    """Integrated autocorrelation time by pairwise blocking (the published procedure with the
    reference's lag rule and block-edge window), one row."""
    x = series.astype(np.float64)
    n = x.size
    lag = max(10, min(n // 5, wgs, 64))
    mu = x.mean()
    m = x - mu

    def one(m, lag):
        n = m.size
        b = min(wgs, n)
        t = np.arange(n - lag)
        acc = np.zeros(n - lag)
        for q in range(1, lag + 1):
            u = t + q
            inside = u < (t // b + 1) * b
            acc += np.where(inside & (u + lag >= n), 0.0, m[u])
        xt = m[:n - lag]
        return float(np.sum(xt * xt)), float(np.sum(xt * (xt + 2.0 * acc)))

    c0, d = one(m, lag)
    first, tau, lag2, stride = c0, d / c0, lag, 1
    while 10 < lag2 and lag2 < 5.0 * tau:
        h = m.size // 2
        m = m[0:2 * h:2] + m[1:2 * h:2]
        lag2 = lag if lag * 5 < h else max(h // 5, 10)
        prev = c0
        stride *= 2
        c0, d = one(m, lag2)
        tau = d / prev
    scale = stride * (m.size - lag2)
    return d * (n - lag) / (scale * first), mu, math.sqrt(d / (scale * n))


def exact(case, seed):
    kind = case["kind"]
    if kind == "logistic":
        if 2.0 * case["rows"] * case["features"] * case["walkers"] > 1.2e12:
            return None
        f = case["features"]
        params, pos = _logistic_inputs(case, seed)
        rows = params[:-1].view(case["rows"], f + 1)
        b = pos.double()
        acc = -(b * b).sum(1) / 50.0
        step = max(1, (1 << 29) // case["walkers"])
        for r0 in range(0, case["rows"], step):
            blk = rows[r0:r0 + step].double()
            eta = blk[:, :f] @ b.T
            acc += (blk[:, f:] * eta - eta.clamp(min=0.0) - torch.log1p(torch.exp(-eta.abs()))).sum(0)
        return acc
    if kind == "data":
        x = _data_matrix(case, seed)
        v = x.double()
        mu = v.mean(0)
        return dict(mean=mu, variance=((v - mu) ** 2).mean(0),
                    limits=torch.stack([v.min(0).values, v.max(0).values], 1), pdf=None, ranks=None)
    if kind == "density":
        y, x = _density_inputs(case, seed)
        y = torch.from_numpy(y).cuda().double()
        x = torch.from_numpy(x).cuda().double()
        ld = torch.zeros(x.shape[0], dtype=torch.float64, device="cuda")
        for v in y:
            ld += -((v - x[:, 0]) ** 2) / (2.0 * x[:, 1] ** 2) - torch.log(x[:, 1]) - LOG_SQRT_2PI
        return dict(log_density=ld, evidence=torch.exp(ld).mean())
    if kind == "acor":
        r = [_acor64(row) for row in _acor_series(case, seed)]
        return dict(tau=np.array([v[0] for v in r]), mean=np.array([v[1] for v in r]),
                    sigma=np.array([v[2] for v in r]))
    return None
