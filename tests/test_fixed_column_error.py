"""The fixed-point velocity column (csrc/joker_fixed.cuh) against the same
formulas in doubles (csrc/joker_math.cuh, OrbitF64), both compiled for the host
and compared with long double values: wherever as_exact() lets an orbit take the
fixed-point form, its rms error near pericentre is no larger.

Long double carries at least 11 bits more than a double, in the phase and in
the solve, so that its own error stays below 2^-11 of the doubles'."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "thejoker_gb300", "csrc")
SOURCE = r"""
#include <random>
#include "joker_fixed.cuh"
using namespace joker::fx;
typedef long double ld;
static const ld PI = 3.141592653589793238462643383279502884L;

static double root(double x, double e) {                  // E - e sin E = x
    double E = std::fmin(x + e, (double)PI);
    for (int i = 0; i < 60; ++i) {
        const double f = E - e * sin(E) - x, f1 = 1 - e * cos(E), f2 = e * sin(E);
        const double n = E - 2 * f * f1 / std::fmax(2 * f1 * f1 - f * f2, 1e-30);
        const double c = std::fmin(std::fmax(n, x), x + e);
        if (c == E) break;
        E = c;
    }
    return E;
}
static ld exact(double dt, double P, double e, double om, double M0) {
    ld M = 2 * PI * ((ld)dt / P) - (ld)M0;
    M -= 2 * PI * rintl(M / (2 * PI));
    const ld x = fabsl(M);
    ld E = root((double)x, e);
    for (int i = 0; i < 4; ++i) {
        const ld f = E - e * sinl(E) - x, f1 = 1 - e * cosl(E), f2 = e * sinl(E);
        E -= 2 * f * f1 / (2 * f1 * f1 - f * f2);
    }
    if (M < 0) E = -E;
    const ld c = cosl(E), den = 1 - e * c;
    return cosl(om) * ((c - e) / den + e) -
           sinl(om) * sqrtl((1 - (ld)e) * (1 + (ld)e)) * sinl(E) / den;
}

// sin and cos of k/128 + r as sincos_f32arg and sincos_f64_table form them
static void node(int k, double r, double &s, double &c) {
    const double ts = sin(k / 128.0), tc = cos(k / 128.0), r2 = r * r;
    const double sr = fma(r * r2, fma(r2, 1.0 / 120.0, -1.0 / 6.0), r);
    const double cm1 = r2 * fma(r2, 1.0 / 24.0, -0.5);
    s = fma(ts, cm1, fma(tc, sr, ts));
    c = fma(tc, cm1, fma(-ts, sr, tc));
}
static float starter(float x, float e, float ome, float a1) {
    const float PIf = 3.14159265358979f, PI2 = 9.8696044011f;
    const float alpha = fmaf(a1, PIf - x, 3 * PI2 / (PI2 - 6));
    const float d = fmaf(alpha, e, 3 * ome), x2 = x * x, ad = alpha * d;
    const float q = fmaf(ad, 2 * ome, -x2), r = x * fmaf(ad, fmaf(3, d, -3 * ome), x2);
    const float w = exp2f(0.6666667f * log2f(sqrtf(fmaf(q * q, q, r * r)) + r));
    const float den = fmaf(w, w + q, q * q);
    return fmaf(x, den, 2 * r * w) / (den * d);
}
static double doubles(double dt, double P, double e, double om, double M0) {
    const double T = 6.283185307179586476925, IT = 0.15915494309189533577;
    const double HI = 6.283185307179586, LO = 2.4492935982947064e-16;
    double M = fma(dt, T / P, -M0);
    const double n = rint(M * IT);
    M = fma(-n, LO, fma(-n, HI, M));
    const double x = fabs(M);
    const float a1 = 1.6f * 3.14159265358979f / (9.8696044011f - 6) / (1 + (float)e);
    const float E1 = starter((float)x, (float)e, (float)(1 - e), a1);
    const int k = (int)rintf(E1 * 128);
    double s1, c1;
    node(k, (double)fmaf((float)k, -0.0078125f, E1), s1, c1);
    const double f2 = e * s1, f3 = e * c1, f0 = ((double)E1 - x) - f2, i1 = 1 / (1 - f3);
    const double u = -f0 * i1, t2 = f2 * i1, t3 = f3 * i1, t22 = t2 * t2;
    const double c3 = fma(t22, 0.5, t3 * (-1.0 / 6)), c4 =
        t2 * fma(t22, -0.625, fma(t3, 5.0 / 12, 1.0 / 24));
    const double d = u * fma(u, fma(u, fma(u, c4, c3), -0.5 * t2), 1.0), dd = d * d;
    const double cm1 = dd * fma(dd, 1.0 / 24, -0.5), sd = d * fma(dd, -1.0 / 6, 1.0);
    double sE = fma(s1, cm1, fma(c1, sd, s1));
    const double cE = fma(c1, cm1, fma(-s1, sd, c1));
    if (M < 0) sE = -sE;
    const double nr = rint(om * IT), ox = fma(-nr, LO, fma(-nr, HI, om));
    const int ko = (int)rintf((float)fabs(ox) * 128);
    double sw, cw;
    node(ko, fma((double)ko, -0.0078125, fabs(ox)), sw, cw);
    if (ox < 0) sw = -sw;
    const double B = -sw * sqrt((1 - e) * (1 + e)), D = e * cw;
    return fma(fma(cw, cE, fma(B, sE, -D)), 1 / fma(-e, cE, 1.0), D);
}

// Squared errors of n draws with 1 - e in [o0, o1] and span / P in [T0, T1], the
// epoch within ten widths (1 - e)^1.5 of pericentre; of those taken.
extern "C" int errors(int n, int seed, double o0, double o1, double T0, double T1, double *out) {
    std::mt19937_64 g(seed);
    auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    int taken = 0;
    out[0] = out[1] = 0;
    for (int i = 0; i < n; ++i) {
        const double ome = o0 * pow(o1 / o0, U(0, 1)), e = 1 - ome, span = exp2(U(0, 12));
        const double P = span / (T0 * pow(T1 / T0, U(0, 1))), om = U(0, 6.28);
        const int tsh = 62 - (ilogb(span) + 1);
        const double dt = ldexp(rint(ldexp(U(0, span), 30)), -30);
        const double M = pow(ome, 1.5) * pow(10, U(-2, 1)) * (g() & 1 ? 1 : -1);
        const double M0 = fmod(2 * (double)PI * (dt / P) - M + 2 * (double)PI, 2 * (double)PI);
        Orbit o;
        if (!as_exact(tsh, P, e) || !o.init(tsh, 0, P, e, om, M0)) continue;
        const ld want = exact(dt, P, e, om, M0);
        const ld f = ldexpl((ld)o.column((uint64_t)ldexp(dt, tsh)), -61) - want;
        const ld d = (ld)doubles(dt, P, e, om, M0) - want;
        out[0] += (double)(f * f);
        out[1] += (double)(d * d);
        ++taken;
    }
    return taken;
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("column")
    src, so = str(d / "c.cc"), str(d / "c.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    CSRC, src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    dbl = ctypes.c_double
    lib.errors.argtypes = [ctypes.c_int, ctypes.c_int, dbl, dbl, dbl, dbl,
                           ctypes.POINTER(dbl)]
    return lib


@pytest.mark.parametrize("q", [-12, -7, -5, -4, -3, -2, -1, 0, 2, 8])
def test_no_less_exact_than_doubles(host, q):
    out = (ctypes.c_double * 2)()
    n = 4000
    for k in range(10):
        o0 = max(2.0 ** -(k + 1), 0.0010001)
        taken = host.errors(n, 100 * k + q + 20, o0, 2.0 ** -k, 2.0 ** q, 2.0 ** (q + 1), out)
        if taken > n // 20:
            assert out[0] <= out[1], (k, taken, np.sqrt(out[0] / out[1]))
        # what the fixed-point form is for: periods up to the span (the rule
        # knows both to a power of two), and ordinary eccentricities at any period
        if q >= 0 or k < 3:
            assert taken == n
