"""The plain form's kernels where the wait for the staged params gives up: run on the host, one
thread, with the device source's own text and stand-ins for the wait and the density.

A density must not be evaluated then (what it reads may be anything, lengths and offsets
included), and no finite value may come of it.
"""
import ctypes as C
import os
import re
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

SRC = os.path.join(ROOT, "bayadera_gb300", "csrc", "device", "bay_stretch.cuh")

STUBS = r"""
#include <cmath>
#include <cstring>
#include <cstdint>
#define __device__
#define __forceinline__ inline
#define __shared__ static
#define DIM 2
#define BAY_CTA 1
struct dim3_ { unsigned int x; };
static const dim3_ threadIdx = {0}, blockIdx = {0}, blockDim = {1}, gridDim = {1};
static inline void __syncthreads() {}
static inline float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
struct bay_plain_sync { unsigned long long bar; };
static bool lands;            // whether the wait succeeds
static int evaluated;         // densities evaluated
template <bool STAGED> void bay_stage_begin(bay_plain_sync*, const float*, unsigned int) {}
template <bool STAGED> bool bay_stage_wait(bay_plain_sync*, unsigned int* status) {
    if (!lands && status) *status |= 1u;
    return lands;
}
template <bool STAGED>
float bay_density(unsigned int, unsigned int, const float* params, const float* x) {
    ++evaluated;
    return -(x[0] * x[0] + x[1] * x[1]) * params[0];
}
"""

POINTS = r"""
extern "C" void set_lands(int v) { lands = v != 0; evaluated = 0; }
extern "C" int count() { return evaluated; }
extern "C" double evidence(unsigned long long n, const float* params, const float* x) {
    double part = -1.0;
    bay_points_sum<true>(n, 0u, 1u, params, x, &part);
    return part;
}
extern "C" void density(unsigned long long n, const float* params, const float* x, float* out) {
    bay_points_density<true>(n, 0u, 1u, params, x, out, 1u);
}
"""


def function(text, name):
    """The template function `name` of the source, without its inline assembly."""
    at = text.index(name + "(")
    start = text.rindex("template <", 0, at)
    end = text.index("\n}\n", at) + 3
    body = re.sub(r"asm(?: volatile)?\(.*?\);", ";", text[start:end], flags=re.S)
    return body.replace("unsigned int ncta, rank;", "unsigned int ncta = 1u, rank = 0u;")


def host_library(tmp_path, names, tail, stubs=""):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    text = open(SRC).read()
    src, lib = tmp_path / "host.cpp", tmp_path / "host.so"
    src.write_text(STUBS + stubs + "".join(function(text, n) for n in names) + tail)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fno-strict-aliasing", "-shared", "-fPIC", "-w", str(src),
                    "-o", str(lib)], check=True)
    return C.CDLL(str(lib))


@pytest.mark.parametrize("n", [0, 1, 5])
def test_points_are_not_evaluated_and_give_nan_where_the_params_did_not_land(tmp_path, n):
    lib = host_library(tmp_path, ["bay_points_density", "bay_points_sum"], POINTS)
    lib.evidence.restype = C.c_double
    params, x = (C.c_float * 1)(0.5), (C.c_float * 10)(*range(10))
    want = [C.c_float(0.0).value + 2.718281828459045 ** (-0.5 * ((2 * i) ** 2 + (2 * i + 1) ** 2))
            for i in range(n)]
    for lands in (1, 0):
        out = (C.c_float * 5)(*[7.0] * 5)
        lib.set_lands(lands)
        e = lib.evidence(C.c_ulonglong(n), params, x)
        lib.density(C.c_ulonglong(n), params, x, out)
        assert lib.count() == (2 * n if lands else 0)
        if lands:
            assert e == pytest.approx(sum(want), rel=1e-6)
            assert list(out[:n]) == pytest.approx(want, rel=1e-5)
        else:
            assert e != e and all(v != v for v in out[:n])
        assert list(out[n:]) == [7.0] * (5 - n)


MOVE_STUBS = r"""
#include <cstddef>
#define BAY_SUM_CHUNK 64
struct bay_u4 { unsigned int x, y, z, w; };
struct ctl_ { unsigned int step[2], seed[2]; float a, beta; unsigned int status; };
struct bay_stretch_params {
    float* xs; float* logfn; const float* params; ctl_* ctl;
    unsigned int K, half, step_off, params_len;
    unsigned long long data_len;
};
static bay_u4 bay_philox4x32_10(bay_u4 c, unsigned int, unsigned int) { return c; }
static float bay_u01(unsigned int) { return 0.5f; }
static float bay_stretch_z(float, float) { return 0.5f; }
static unsigned int bay_partner(float, unsigned int) { return 0u; }
static float bay_partner_coord(const float* S, unsigned int, unsigned int j, int i) { return S[j * DIM + i]; }
static float bay_beta(const bay_stretch_params&) { return 1.0f; }
static bool bay_accept(float, float, float, float, float) { return true; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmaf_rn(float a, float b, float c) { return a * b + c; }
#undef BAY_CTA
#define BAY_CTA 32
static float kept[DIM];
static bool counted;
static void bay_accu_epilogue(const bay_stretch_params&, bool accepted, bool, const float* mine,
                              float (*)[BAY_SUM_CHUNK], unsigned int, unsigned int, unsigned int, unsigned int) {
    counted = accepted;
    for (int i = 0; i < DIM; ++i) kept[i] = mine[i];
}
"""

MOVE = r"""
extern "C" void set_lands(int v) { lands = v != 0; evaluated = 0; }
extern "C" int count() { return evaluated; }
extern "C" unsigned int move(int accu, float* xs, float* logfn, const float* params, float* mine) {
    ctl_ ctl = {};
    ctl.a = 2.0f;
    bay_stretch_params P = {xs, logfn, params, &ctl, 1u, 0u, 0u, 1u, 0ull};
    counted = false;
    if (accu) bay_stretch_plain<true, true>(P);
    else bay_stretch_plain<false, true>(P);
    for (int i = 0; i < DIM; ++i) mine[i] = kept[i];
    return ctl.status | (counted ? 2u : 0u);
}
"""


@pytest.mark.parametrize("accu", [0, 1])
def test_moves_are_rejected_unevaluated_where_the_params_did_not_land(tmp_path, accu):
    lib = host_library(tmp_path, ["bay_stretch_plain"], MOVE,
                       MOVE_STUBS)
    params = (C.c_float * 1)(0.5)
    for lands in (1, 0):
        xs, logfn, mine = (C.c_float * 4)(3.0, 4.0, 1.0, 2.0), (C.c_float * 2)(-9.0, -9.0), (C.c_float * 2)()
        lib.set_lands(lands)
        got = lib.move(accu, xs, logfn, params, mine)
        assert lib.count() == lands
        moved = [2.0, 3.0] if lands else [3.0, 4.0]
        assert list(xs) == moved + [1.0, 2.0] and logfn[0] == (-6.5 if lands else -9.0)
        if accu:
            assert list(mine) == moved
        assert got == ((2 if accu else 0) if lands else 1)
