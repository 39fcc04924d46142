"""The erf of the 4-parameter Gaussian fit (Abramowitz & Stegun 7.1.26) takes the reciprocal of 1 + p |x| from the
special-function unit, which is off by up to 1 ulp. Compiled here for the host with a reciprocal that is off by that
much in either direction, it has to give what the rounded quotient gives: one refinement leaves an error of 2^-47
relative before the last rounding, so all but about 1e-6 of the quotients round alike.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np

SRC = Path(__file__).resolve().parent.parent / "qtrk_b200" / "csrc" / "device_common.cuh"
HOST = """
#include <cmath>
#define __device__
#define __forceinline__ inline
static int g_ulps = 0;
static float rcp(float x)
{
    float r = 1.0f / x;
    for (int k = 0; k < (g_ulps < 0 ? -g_ulps : g_ulps); k++) r = nextafterf(r, g_ulps < 0 ? -INFINITY : INFINITY);
    return r;
}
%s
extern "C" void run(const float *x, const float *e, float *y, int n, int ulps)
{
    g_ulps = ulps;
    for (int i = 0; i < n; i++) y[i] = erf_as(x[i], e[i]);
}
"""


def test_the_reciprocal_is_as_good_as_the_quotient(tmp_path):
    text = SRC.read_text()
    start = text.index("__device__ __forceinline__ float erf_as(")
    body = text[start:text.index("\n}\n", start) + 3]
    (tmp_path / "erf.cpp").write_text(HOST % body)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-mfma", "-shared", "-fPIC", "-o", str(tmp_path / "erf.so"),
                    str(tmp_path / "erf.cpp")], check=True)
    lib = C.CDLL(str(tmp_path / "erf.so"))
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-6, 6, 200_000), rng.normal(size=200_000), [0.0, -0.0, 1e30, -1e30, 3e38, -3e38,
                                                                               np.inf, -np.inf]]).astype(np.float32)
    with np.errstate(over="ignore"):
        e = np.exp(-x.astype(np.float64) ** 2).astype(np.float32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    y = []
    for ulps in (0, 1, -1):
        out = np.empty_like(x)
        lib.run(p(x), p(e), p(out), len(x), ulps)
        y.append(out)
    for off in y[1:]:
        assert np.mean(off != y[0]) < 1e-4 and np.abs(off - y[0]).max() < 2e-7
        assert np.array_equal(off[-8:], y[0][-8:])
    nan = np.array([np.nan], np.float32)
    out = np.zeros(1, np.float32)
    lib.run(p(nan), p(nan), p(out), 1, 0)
    assert np.isnan(out[0])
