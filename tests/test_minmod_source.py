"""The limiter of the CUDA source itself (euler_state.cuh, compiled for the
host with the few device intrinsics it uses spelled out), against the
reference's formula 0.5 (sgn(a) + sgn(b)) min(|a|, |b|) (real.h:63-65) and its
three-argument form (vector.h:195-202): equal values over a grid of ordinary,
tiny, huge and special numbers (zeros may differ in sign)."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import PKG, ROOT

HARNESS = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __host__
#define __forceinline__ inline
#define __restrict__
using std::copysign;
using std::fabs;
using std::sqrt;
using std::pow;
static inline long long __double_as_longlong(double a) { long long r; std::memcpy(&r, &a, 8); return r; }
static inline int __double2hiint(double a) { return (int)(__double_as_longlong(a) >> 32); }
static inline unsigned __float_as_uint(float a) { unsigned r; std::memcpy(&r, &a, 4); return r; }
static inline int __float_as_int(float a) { int r; std::memcpy(&r, &a, 4); return r; }
static inline float fabsf_(float a) { return std::fabs(a); }
#include "euler_state.cuh"
extern "C" {
void two_d(long n, const double* a, const double* b, double* r) {
    for (long i = 0; i < n; i++) r[i] = amr::minmod2(a[i], b[i]);
}
void two_f(long n, const float* a, const float* b, float* r) {
    for (long i = 0; i < n; i++) r[i] = amr::minmod2(a[i], b[i]);
}
void theta_d(long n, const double* a, const double* b, double t, double* r) {
    for (long i = 0; i < n; i++) r[i] = amr::minmod_theta(a[i], b[i], t);
}
}
"""


def reference(a, b):
    sgn = lambda x: np.where(x > 0, 1.0, np.where(x < 0, -1.0, 0.0)).astype(a.dtype)
    fa, fb = np.abs(a), np.abs(b)
    return a.dtype.type(0.5) * (sgn(a) + sgn(b)) * np.where(fa > fb, fb, fa)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("minmod")
    src = d / "h.cpp"
    src.write_text(HARNESS)
    so = str(d / "h.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-fPIC", "-shared", "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(ROOT, "include"), str(src), "-o", so], check=True)
    return ctypes.CDLL(so)


def grid(dt):
    rng = np.random.default_rng(3)
    f = np.finfo(dt)
    v = [0.0, f.tiny, f.smallest_subnormal, 1.0, 1.0 + f.eps, 0.75, 1e10, f.max, np.inf, np.nan]
    v = np.array(v + [-x for x in v] + list(rng.standard_normal(200) * 10.0 ** rng.uniform(-30, 30, 200)), dt)
    a, b = np.meshgrid(v, v)
    return np.ascontiguousarray(a.ravel()), np.ascontiguousarray(b.ravel())


def pointers(*arrays):
    return [x.ctypes.data_as(ctypes.c_void_p) for x in arrays]


@pytest.mark.parametrize("dt,name", [(np.float64, "two_d"), (np.float32, "two_f")])
def test_minmod(lib, dt, name):
    a, b = grid(dt)
    got = np.empty_like(a)
    getattr(lib, name)(ctypes.c_long(a.size), *pointers(a, b, got))
    with np.errstate(all="ignore"):
        assert np.array_equal(got, reference(a, b), equal_nan=True)


@pytest.mark.parametrize("theta", [1.0, 1.3, 2.0])
def test_minmod_theta(lib, theta):
    up, um = grid(np.float64)
    got = np.empty_like(up)
    lib.theta_d(ctypes.c_long(up.size), *pointers(up, um), ctypes.c_double(theta), *pointers(got))
    with np.errstate(all="ignore"):
        want = reference(theta * up, reference(theta * um, 0.5 * (up + um)))
    assert np.array_equal(got, want, equal_nan=True)
