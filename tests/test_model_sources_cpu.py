"""Which plain-form sources get kernels with their params in shared memory (named _s): plain C and
arithmetic, not what names an address space or has shared memory of its own.  From ptxas' report,
no device needed."""
import re

import pytest

BASE = """
extern "C" {
%(before)s
inline REAL density(const uint32_t data_len, const uint32_t params_len, const REAL* params,
                    const uint32_t dim, const REAL* x) {
    REAL acc = 0.0f;
    for (uint32_t i = 0; i < data_len; ++i) { const REAL d = x[0] - %(load)s; acc -= d * d; }
    return acc;
}
}
"""

STAGED = {
    "plain": ("", "params[i]"),
    "vector": ("", "reinterpret_cast<const float2*>(params)[i / 2u].x"),
    "memcpy": ("inline REAL get(const REAL* p) { REAL v; memcpy(&v, p, 4); return v; }", "get(params + i)"),
    "arithmetic": ("", "__fmul_rn(__expf(params[i]), __uint2float_rn(__popc(1'000u * i)))"),
    "qualifiers": ("static __device__ __forceinline__ REAL get(const REAL* __restrict__ p) { return *p; }",
                   "get(params + i)"),
    "comments": ("// __ldg(p), asm\n/* __shared__\n ## */ static const char* const name = \"__ldg asm ##\";",
                 "params[i]"),
    "include": ("}\n#include <stdint.h>\n#  include <cstdint>\nextern \"C\" {", "params[i]"),
    "inner underscores": ("inline REAL get__asm(const REAL* p) { return *p; }", "get__asm(params + i)"),
}
GLOBAL = {
    "ldg": ("", "__ldg(params + i)"),
    "ldcg": ("", "__ldcg(params + i)"),
    "ldcs in a macro": ("#define LOAD(p) __ldcs(p)", "LOAD(params + i)"),
    "asm": ("inline REAL get(const REAL* p) { REAL v; asm(\"ld.global.f32 %%0, [%%1];\" : \"=f\"(v) : \"l\"(p));"
            " return v; }", "get(params + i)"),
    "space test": ("", "(__isGlobal(params) ? params[i] : 0.0f)"),
    "conversion": ("", "(REAL)(uint32_t)(__cvta_generic_to_global(params) != 0)"),
    "pasted": ("#define LOAD(name, p) __ld##name(p)", "LOAD(g, params + i)"),
    "pasted by digraph": ("#define LOAD(name, p) __ld%%:%%:name(p)", "LOAD(g, params + i)"),
    "spliced": ("", "__l\\\ndg(params + i)"),
    "own shared memory": ("__shared__ REAL table[64];", "params[i] + table[0]"),
    "raw string": ("static const char* const name = R\"(\")\"; // \"", "params[i]"),
}


@pytest.fixture(scope="module")
def native():
    from bayadera_gb300 import _native, build
    build.build()
    return _native


def staged(model, monkeypatch, capfd, tag):
    """Whether the model's plain form has the staged kernels, the unstaged ones in any case."""
    from bayadera_gb300.engine import check_model
    monkeypatch.setenv("BAY_PTXAS_VERBOSE", "1")
    model.sources = model.sources + ["// %s" % tag]        # not in the process's cache
    capfd.readouterr()
    check_model(model, "plain")
    report = capfd.readouterr().err
    names = ["bay_stretch_bare", "bay_stretch_accu", "bay_logfn_all", "bay_points_logfn", "bay_points_evidence"]
    assert all("'%s'" % n in report for n in names)
    have = ["'%s_s'" % n in report for n in names]
    assert len(set(have)) == 1
    return have[0]


@pytest.mark.parametrize("name", list(STAGED) + list(GLOBAL))
def test_sources_that_may_have_their_params_in_shared_memory(native, name, monkeypatch, capfd):
    from bayadera_gb300 import models as M
    before, load = (STAGED.get(name) or GLOBAL[name])
    src = BASE % {"before": before.replace("%%", "%"), "load": load}
    m = M.device_distribution_model(src, name="density", logpdf="density", dimension=1, params_size=0)
    assert staged(m, monkeypatch, capfd, "sources " + name) == (name in STAGED)


def test_the_built_in_models_may(native, monkeypatch, capfd):
    from bayadera_gb300 import models as M
    dist = M.distribution_models()
    models = list(dist.values()) + [M.gaussian_posterior_model(), M.mvn_precision_model(3), M.logistic_model(3),
                                    M.robust_t_model(3), M.hierarchical_model(2), M.hierarchical_rows_model(2)]
    models += [M.device_posterior_model(dist["gaussian"], "post_" + k, v)
               for k, v in M.likelihood_models().items()]
    for m in models:
        assert staged(m, monkeypatch, capfd, "built in"), m.name


def test_a_gemm_source_with_shared_memory_of_its_own_can_be_launched(native, monkeypatch, capfd):
    """The streamed propose kernel keeps 8 rows of 1,500 coordinates in static shared memory, which
    leaves no room in the 48 KB of a launch for the source's: such a source's rows are read from
    global memory."""
    from bayadera_gb300 import models as M
    from bayadera_gb300.engine import check_model
    src = M.get_source("mvn_precision") + """
extern "C" {
inline void own_prep(const REAL* hyper, const uint32_t hyper_len, const uint32_t dim, const REAL* x, REAL* prep) {
    __shared__ volatile REAL table[2048];
    table[threadIdx.x] = x[0];
    prep[0] = table[threadIdx.x];
}
}
"""
    gemm = dict(M.mvn_precision_model(8).gemm, prep="own_prep", features=8, ld=8, rows=8)
    m = M.device_distribution_model(src, name="own", dimension=1500, params_size=64,
                                    logpdf="mvn_precision_logpdf", gemm=gemm)
    monkeypatch.setenv("BAY_PTXAS_VERBOSE", "1")
    capfd.readouterr()
    check_model(m, "gemm")
    used = re.findall(r"entry function '(bay_gemm_propose_\w+)'.*?(\d+) bytes smem", capfd.readouterr().err, re.S)
    assert len(used) == 3 and all(int(n) <= 48 * 1024 for _, n in used), used
