"""The device code's own elementary functions on the CPU: the sources of
fz_physics.cuh and fz_layer2.cuh compiled for the host, their PTX primitives
(packed FP32 operations, approximate reciprocals) replaced by host ones of the
same rounding, or of the hardware's error where it is approximate.

Bounds: rcp_d 2.3e-16 and exp_tab 4e-16 of the value (an ulp is up to 2.2e-16),
the FP32 exponential 2e-7 of e^x and of e^x - 1.  The operator's functions are
compared with their power series in FP64; a root's quotient loses some 1e-6 /
theta (six roundings of 6e-8 and their factors).
"""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "firtez-dz_b200", "csrc")

SHIM = r"""
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
using std::max; using std::min; using std::isnan;
#define __device__
#define __constant__ static const
#define __forceinline__ inline
static inline int __float_as_int(float x) { int i; memcpy(&i, &x, 4); return i; }
static inline float __int_as_float(int i) { float x; memcpy(&x, &i, 4); return x; }
static inline int64_t bits(double x) { int64_t i; memcpy(&i, &x, 8); return i; }
static inline int __double2loint(double x) { return (int)bits(x); }
static inline int __double2hiint(double x) { return (int)(bits(x) >> 32); }
static inline double __hiloint2double(int h, int l) {
  int64_t i = ((int64_t)h << 32) | (uint32_t)l; double x; memcpy(&x, &i, 8); return x; }
static inline double __dmul_rn(double a, double b) { return a * b; }
"""

# device function -> host body
BODIES = {
    r"double rcp_d\(double y\)": "double r = (1.0 / y) * (1.0 + 9.0e-7); const double e = fma(-y, r, 1.0);"
                                 " return fma(r, fma(e, e, e), r);",
    r"float rcp_a\(float y\)": "return 1.0f / y;",
    r"float rsqrt_a\(float y\)": "return 1.0f / sqrtf(y);",
    r"float min_nan\(float x, float y\)": "return isnan(x) || isnan(y) ? NAN : fminf(x, y);",
    r"F2 f2\(float a, float b\)": "F2 r; float v[2] = {a, b}; memcpy(&r.v, v, 8); return r;",
    r"void f2_get\(F2 x, float& a, float& b\)": "float v[2]; memcpy(v, &x.v, 8); a = v[0]; b = v[1];",
    r"F2 fma2\(F2 a, F2 b, F2 c\)": "float x[2], y[2], z[2]; memcpy(x, &a.v, 8); memcpy(y, &b.v, 8);"
                                    " memcpy(z, &c.v, 8); return f2(fmaf(x[0], y[0], z[0]), fmaf(x[1], y[1], z[1]));",
    r"F2 operator\*\(F2 a, F2 b\)": "float x[2], y[2]; memcpy(x, &a.v, 8); memcpy(y, &b.v, 8);"
                                    " return f2(x[0] * y[0], x[1] * y[1]);",
    r"F2 operator\+\(F2 a, F2 b\)": "float x[2], y[2]; memcpy(x, &a.v, 8); memcpy(y, &b.v, 8);"
                                    " return f2(x[0] + y[0], x[1] + y[1]);",
}

MAIN = r"""
using namespace fzd;
extern "C" {
void t_rcp(int n, const double* y, double* r) { for (int i = 0; i < n; ++i) r[i] = rcp_d(y[i]); }
void t_exp(int n, int form, const double* x, double* r) {
  double tab[32];
  for (int j = 0; j < 32; ++j) tab[j] = exp2(j / 32.0);
  for (int i = 0; i < n; ++i)
    r[i] = form == 0 ? exp_tab<false>(x[i], tab) : form == 1 ? exp_tab<true>(x[i], tab) : exp_any(x[i], tab);
}
static void put(F2 x, float* o, int i) { f2_get(x, o[i], o[i + 1]); }
void t_expf(int n, const float* x, float* e, float* em1) {
  for (int i = 0; i < n; i += 2) {
    const ExpF2 p = exp_parts2(f2(x[i], x[i + 1]));
    put(p.exp(), e, i);
    put(p.expm1(), em1, i);
  }
}
void t_evol(int n, const float* d, const float* e, float* v) {   // v[14][n]
  for (int i = 0; i < n; i += 2) {
    const F2 a = f2(d[i], d[i + 1]), b = f2(e[i], e[i + 1]);
    const EvolABG2 p = evol_abg2(a, b);
    const EvolD2 q = evol_d2(a, b);
    const F2 o[14] = {p.am, p.al, p.be, p.ga, q.am, q.al, q.be, q.ga, q.al_d, q.al_e, q.be_d, q.be_e, q.ga_d, q.ga_e};
    for (int k = 0; k < 14; ++k) put(o[k], v + (size_t)k * n, i);
  }
}
// layers t[7][n] (I, Q, U, V, rho Q, U, V), changes dt[7][n], vectors w[4][n]
// -> O w and its change, out[8][n]
void t_resp(int n, const float* t, const float* dt, const float* w, float* out) {
  for (int i = 0; i < n; i += 2) {
    auto g = [&](const float* p, int k) { return f2(p[(size_t)k * n + i], p[(size_t)k * n + i + 1]); };
    LayerD2 L;
    F2 x[3], y[3], ww[4], o[4];
    for (int k = 0; k < 3; ++k) L.t[k] = g(t, 1 + k), L.r[k] = g(t, 4 + k), x[k] = g(dt, 1 + k), y[k] = g(dt, 4 + k);
    for (int k = 0; k < 4; ++k) ww[k] = g(w, k);
    layer_d2(L, g(t, 0));
    Resp2 R;
    resp_w(L, ww, R);
    resp_dir(L, R, g(dt, 0), x, y, o);
    for (int k = 0; k < 4; ++k) put(R.Ow[k], out + (size_t)k * n, i), put(o[k], out + (size_t)(4 + k) * n, i);
  }
}
}
"""


def _function(src, sig):
    """(start, end) of the function whose declaration matches sig."""
    m = re.search(r"^(template <[^\n]*\n)?__device__ __forceinline__ " + sig + r" \{", src, re.M)
    assert m, sig
    i, depth = m.end(), 1
    while depth:
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        i += 1
    return m.start(), i


def _host_source():
    phys = open(os.path.join(CSRC, "fz_physics.cuh")).read()
    lay = open(os.path.join(CSRC, "fz_layer2.cuh")).read()
    parts = re.findall(r"^__constant__ double EXP_C.*?;\n|^constexpr float [^;]*;\n", phys, re.M | re.S)
    for sig in (r"double rcp_d\(double y\)", r"double exp_tab\([^)]*\)", r"double exp_any\([^)]*\)",
                r"float rcp_a\(float y\)", r"float rsqrt_a\(float y\)", r"float min_nan\(float x, float y\)"):
        a, b = _function(phys, sig)
        parts.append(phys[a:b] + "\n")
    src = "namespace fzd {\n" + "".join(parts) + "}\n" + re.sub(r"^#(include|pragma once).*\n", "", lay, flags=re.M)
    for sig, body in BODIES.items():
        a, b = _function(src, sig)
        head = src[a:b].split("{", 1)[0]
        src = src[:a] + head + "{ " + body + " }" + src[b:]
    assert "asm" not in src.replace("asm volatile", "asm")
    return SHIM + src + MAIN


@pytest.fixture(scope="module")
def dev(tmp_path_factory):
    d = tmp_path_factory.mktemp("devmath")
    (d / "m.cpp").write_text(_host_source())
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-o",
                           str(d / "m.so"), str(d / "m.cpp")])
    return ctypes.CDLL(str(d / "m.so"))


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def test_reciprocal(dev):
    rng = np.random.default_rng(0)
    y = np.ldexp(1.0 + rng.random(1 << 16), rng.integers(-400, 400, 1 << 16)) * rng.choice([-1.0, 1.0], 1 << 16)
    r = np.empty_like(y)
    dev.t_rcp(y.size, _ptr(y), _ptr(r))
    err = np.abs(r.astype(np.longdouble) * y - 1)
    assert err.max() <= 2.3e-16


def _exp(dev, form, x):
    r = np.empty_like(x)
    dev.t_exp(x.size, form, _ptr(x), _ptr(r))
    return r


def test_exponential_in_double(dev):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-700, 700, 50000), rng.uniform(-1, 1, 10000), np.ldexp(rng.random(5000), -40),
                        np.arange(-64, 65) * np.log(2) / 64, [0.0, -0.0, 700.0, -700.0]])
    want = np.exp(x.astype(np.longdouble))
    for form in (0, 1, 2):
        assert np.max(np.abs(_exp(dev, form, x) / want - 1)) <= 4e-16, form
    # the form with the cut ends at 2^+-1020 and the next powers, and keeps NaN
    big = np.array([800.0, 1e4, 4e7, -800.0, -1e4, -4e7, np.nan])
    v = _exp(dev, 1, big)
    assert np.all(v[:3] >= 2.0 ** 1020) and np.all(v[3:6] <= 2.0 ** -1019) and np.all(v[3:6] > 0) and np.isnan(v[6])
    # exp_any is exp() outside the table's range
    odd = np.array([704.0, 709.0, 710.0, -744.0, -746.0, 1e10, -1e300, np.inf, -np.inf, np.nan])
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(_exp(dev, 2, odd), np.exp(odd))


def test_exponential_in_single(dev):
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-87, 88, 40000), rng.uniform(-1, 1, 20000), np.ldexp(rng.random(4000), -30)]).astype(np.float32)
    e, m = np.empty_like(x), np.empty_like(x)
    dev.t_expf(x.size, _ptr(x), _ptr(e), _ptr(m))
    assert np.max(np.abs(e / np.exp(x.astype(np.float64)) - 1)) <= 2e-7
    w = np.expm1(x.astype(np.float64))
    assert np.max(np.abs(m - w) / np.abs(w)) <= 2e-7
    # 0 from below 2^-126 to the depths that are cut, large and finite up to 2^21
    lo = np.array([-88.1, -89, -104, -1e3, -1e5, -1e7, -1e9, -9.9e11], dtype=np.float32)
    e, m = np.empty_like(lo), np.empty_like(lo)
    dev.t_expf(lo.size, _ptr(lo), _ptr(e), _ptr(m))
    assert np.all(e == 0) and np.all(m == -1)
    hi = np.array([88.8, 95, 104, 1e3, 1e4, 1e5, 1e6, 2e6], dtype=np.float32)
    e, m = np.empty_like(hi), np.empty_like(hi)
    dev.t_expf(hi.size, _ptr(hi), _ptr(e), _ptr(m))
    assert np.all(np.isfinite(m)) and np.all(m > 1.1e38)
    nan = np.array([np.nan, 1.0], dtype=np.float32)
    e, m = np.empty_like(nan), np.empty_like(nan)
    dev.t_expf(2, _ptr(nan), _ptr(e), _ptr(m))
    assert np.isnan(e[0]) and np.isnan(m[0]) and abs(e[1] - np.e) < 1e-6


def _series(d, e, terms=48):
    """am, al, be, ga and al_d, al_e, be_d, be_e, ga_d, ga_e in FP64: with u1 = x^2
    and u2 = -y^2 the roots of u^2 - d u - e^2, divided differences of the even
    power series, by the recursion of the complete symmetric polynomials h."""
    d, e = d.astype(np.float64), e.astype(np.float64)
    z = np.zeros_like(d)
    h = [z, z + 1.0]            # h_{-1}, h_0 and their derivatives by d and e
    hd, he = [z, z], [z, z]
    p = [z + 2.0, d]
    for _ in range(terms):
        h.append(d * h[-1] + e * e * h[-2])
        hd.append(h[-2] + d * hd[-1] + e * e * hd[-2])
        he.append(2 * e * h[-3] + d * he[-1] + e * e * he[-2])
        p.append(d * p[-1] + e * e * p[-2])
    f = np.cumprod(np.concatenate([[1.0], np.arange(1, 2 * terms + 2, dtype=np.float64)]))
    s = lambda q, k0, c: sum(q[n + k0] / c(n) for n in range(1, terms))   # noqa: E731
    am = 0.5 * sum(p[n] / f[2 * n] for n in range(1, terms))
    al, ald, ale = (q[1] + s(q, 1, lambda n: f[2 * n + 1]) for q in (h, hd, he))
    ga, gad, gae = (s(q, 0, lambda n: f[2 * n]) for q in (h, hd, he))
    b, bd, be_ = (s(q, 0, lambda n: f[2 * n + 1]) for q in (h, hd, he))
    return am, al, -e * b, ga, ald, ale, -e * bd, -b - e * be_, gad, gae


def test_operator_functions_and_their_derivatives(dev):
    """Neighbours of all sizes share a pair: thin beside thick, and degenerate
    ones (d = e = 0) beside both."""
    rng = np.random.default_rng(3)
    n = 20000
    size = np.exp(rng.uniform(np.log(1e-12), np.log(30.0), n))
    size[::7] = 0.0
    a = rng.uniform(0, 2 * np.pi, n)
    d, e = (size * np.cos(a)).astype(np.float32), (size * np.sin(a)).astype(np.float32)
    d[3::11] = 0.0
    e[5::13] = 0.0
    v = np.empty((14, n), dtype=np.float32)
    dev.t_evol(n, _ptr(d), _ptr(e), _ptr(v))
    ref = _series(d, e)
    theta = np.hypot(d.astype(np.float64), 2.0 * e)
    x = np.sqrt(np.maximum(0.5 * (theta + d), 0.0))
    # series up to 1/4 (1/64 beside a thick one), quotients by theta above
    tol = 1e-6 * np.cosh(x) * (1.0 + x) * np.maximum(1.0, 1.0 / np.maximum(theta, 1.0 / 64))
    for i, k in enumerate(range(4)):
        for row in (k, 4 + k):
            assert np.all(np.abs(v[row] - ref[i]) <= tol), (row, np.max(np.abs(v[row] - ref[i]) / tol))
    for i in range(6):
        assert np.all(np.abs(v[8 + i] - ref[4 + i]) <= tol), (i, np.max(np.abs(v[8 + i] - ref[4 + i]) / tol))


def _matrix(t):
    i, q, u, v, a, b, c = t
    return np.array([[i, q, u, v], [q, i, -c, b], [u, c, i, -a], [v, -b, a, i]])


def test_response_of_a_layer(dev):
    """O w and its change for random directions against the matrix exponential
    and its Frechet derivative; a layer that is not finite has none."""
    from scipy.linalg import expm_frechet
    rng = np.random.default_rng(4)
    n = 400
    t = rng.standard_normal((7, n)) * np.exp(rng.uniform(np.log(1e-5), np.log(2.0), n))
    t[:, ::9] = 0.0
    t[4:, 2::9] = np.roll(t[1:4, 2::9], 1, axis=0)          # |eta| = |rho|
    t[0] = 1.2 * np.linalg.norm(t[1:4], axis=0) + 0.05
    dt, w = rng.standard_normal((7, n)), rng.standard_normal((4, n))
    t, dt, w = (np.ascontiguousarray(q, dtype=np.float32) for q in (t, dt, w))
    out = np.empty((8, n), dtype=np.float32)
    dev.t_resp(n, _ptr(t), _ptr(dt), _ptr(w), _ptr(out))
    for i in range(n):
        o, do = expm_frechet(-_matrix(t[:, i].astype(np.float64)), -_matrix(dt[:, i].astype(np.float64)))
        ww = w[:, i].astype(np.float64)
        s = np.linalg.norm(ww) * (1.0 + np.abs(t[:, i]).max())
        assert np.max(np.abs(out[:4, i] - o @ ww)) <= 2e-6 * s, i
        assert np.max(np.abs(out[4:, i] - do @ ww)) <= 1e-5 * s * np.linalg.norm(dt[:, i]), i
    bad = t[:, :8].copy()
    ddt = dt[:, :8].copy()
    bad[:, 1] = np.nan
    bad[0, 2] = np.inf
    bad[5, 4], bad[5, 5] = np.nan, np.nan
    ddt[:, [1, 2, 4, 5]] = np.nan
    w8, o8 = np.ascontiguousarray(w[:, :8]), np.empty((8, 8), dtype=np.float32)
    dev.t_resp(8, _ptr(bad), _ptr(ddt), _ptr(w8), _ptr(o8))
    gap = [1, 2, 4, 5]
    assert np.all(o8[4:, gap] == 0.0)
    np.testing.assert_array_equal(o8[:4, gap], w8[:, gap])
    keep = [0, 3, 6, 7]
    assert np.all(np.isfinite(o8[:, keep])) and np.max(np.abs(o8[:, keep] - out[:, keep])) < 1e-5
