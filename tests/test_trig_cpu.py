"""The displacement's sine and the adjoint's cosine (mp_trig.cuh, compiled for
the host with the same rounded operations): the short forms equal the general
ones bit for bit over their range, and the cosine keeps its accuracy."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "micropolis_gb300", "csrc")
SOURCE = """
#include <cmath>
#include <cstring>
using std::isfinite;
struct float2 { float x, y; };
static float2 make_float2(float x, float y) { return float2{x, y}; }
static unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
static float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
namespace mp {
static float fmul(float a, float b) { return a * b; }
static float fadd(float a, float b) { return a + b; }
static float fsub(float a, float b) { return a - b; }
static float ffma(float a, float b, float c) { return fmaf(a, b, c); }
static float2 fmul2(float2 a, float2 b) { return float2{a.x * b.x, a.y * b.y}; }
static float2 fadd2(float2 a, float2 b) { return float2{a.x + b.x, a.y + b.y}; }
static float2 ffma2(float2 a, float2 b, float2 c) { return float2{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
static float2 dup2(float a) { return float2{a, a}; }
}
#define MP_TRIG_FN static inline
#include "mp_trig.cuh"
using namespace mp;
extern "C" void run(const float* x, long n, float* sg, float* cg, float* ss, float* cs, float* s2, float* c2) {
    for (long i = 0; i < n; ++i) {
        sg[i] = mp_sinf(x[i]);
        cg[i] = mp_cosf(x[i]);
        ss[i] = sin_small(x[i]);
        cs[i] = cos_small(x[i]);
        s2[i] = i & 1 ? sin2_small(x[i - 1], x[i]).y : sin2_small(x[i], 0.5f).x;
        c2[i] = i & 1 ? cos2_small(x[i - 1], x[i]).y : cos2_small(x[i], 0.5f).x;
    }
}
"""
# positions within 2^18 of the eye's axes, times 22 (displace_is_small)
LARGEST = 22.0 * 2 ** 18


@pytest.fixture(scope="module")
def trig(tmp_path_factory):
    d = tmp_path_factory.mktemp("trig")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unused-function", "-shared", "-fPIC", "-I",
                    CSRC, "-o", str(d / "t.so"), str(d / "t.cpp")], check=True)
    run = ctypes.CDLL(str(d / "t.so")).run

    def call(x):
        x = np.ascontiguousarray(x, np.float32)
        out = [np.empty_like(x) for _ in range(6)]
        p = [a.ctypes.data_as(ctypes.c_void_p) for a in (x, *out)]
        run(p[0], ctypes.c_long(x.size), *p[1:])
        return out
    return call


def _arguments():
    rng = np.random.default_rng(8)
    near = np.arange(-40, 41)[:, None] * (np.pi / 4) + np.arange(-50, 51) * 1e-7   # quadrant borders
    return np.concatenate([rng.uniform(-44, 44, 200001), rng.uniform(-1, 1, 20001) * LARGEST, near.ravel(),
                           10.0 ** rng.uniform(-30, 6.7, 20001), [0.0, -0.0, LARGEST, -LARGEST]]).astype(np.float32)


def test_short_forms_equal_the_general_ones(trig):
    sg, cg, ss, cs, s2, c2 = (a.view(np.uint32) for a in trig(_arguments()))
    assert np.array_equal(ss, sg) and np.array_equal(s2, sg)
    assert np.array_equal(cs, cg) and np.array_equal(c2, cg)


def test_cosine_error(trig):
    """Half an ulp of 1 in the last addition (3.0e-8), two roundings of the
    product r^2 p <= 0.31 before it (3.7e-8), and half an ulp of r <= pi/4
    times the slope there (2.1e-8)."""
    x = np.random.default_rng(9).uniform(-44, 44, 400001).astype(np.float32)
    err = trig(x)[3].astype(np.float64) - np.cos(x.astype(np.float64))
    assert np.abs(err).max() <= 9.0e-8
