"""The fixed-point velocity column (csrc/joker_fixed.cuh) compiled for the
host, against 40-digit values, and the lines where it hands over to doubles.

The bound: the phase is good to 2^-57 of dt / P turns, the last correction is
an FP32 term of order 2^-31 / f' whose relative error is of order 2^-22 / f',
and dm/dE <= 2 / f', with f' = 1 - e cos E >= 1 - e.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "thejoker_gb300", "csrc")
SOURCE = """
#include "joker_fixed.cuh"
using namespace joker::fx;
extern "C" int column(int tsh, int64_t t0, double P, double e, double om, double M0,
                      uint64_t t, int64_t *m) {
    Orbit o;
    if (!o.init(tsh, t0, P, e, om, M0)) return 0;
    *m = o.column(t);
    return o.bad() ? -1 : 1;
}
extern "C" int64_t quotient(int64_t num, int64_t den) { return div61(num, den); }
extern "C" int64_t root(int64_t y) { return sqrt62(y); }
extern "C" uint64_t inverse(uint64_t dn) { return rcp62(dn); }
extern "C" double power(int n, int64_t f) { return exp2_fixed(n, f); }
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed")
    src, so = str(d / "f.cc"), str(d / "f.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    CSRC, src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    i64, u64, dbl = ctypes.c_int64, ctypes.c_uint64, ctypes.c_double
    lib.column.argtypes = [ctypes.c_int, i64, dbl, dbl, dbl, dbl, u64, ctypes.POINTER(i64)]
    lib.quotient.argtypes, lib.quotient.restype = [i64, i64], i64
    lib.root.argtypes, lib.root.restype = [i64], i64
    lib.inverse.argtypes, lib.inverse.restype = [u64], u64
    lib.power.argtypes, lib.power.restype = [ctypes.c_int, i64], dbl
    return lib


def _exact(dt, P, e, om, M0):
    mp = mpmath.mp
    mp.dps = 40
    dt, P, e, om, M0 = (mp.mpf(v) for v in (dt, P, e, om, M0))
    M = 2 * mp.pi * (dt / P) - M0
    M -= 2 * mp.pi * mp.nint(M / (2 * mp.pi))
    x = abs(M)
    lo, hi = x, x + e
    E = min(hi, mp.pi)
    for _ in range(200):
        f = E - e * mp.sin(E) - x
        lo, hi = (lo, E) if f > 0 else (E, hi)
        new = E - f / (1 - e * mp.cos(E))
        new = new if lo <= new <= hi else (lo + hi) / 2
        if abs(new - E) < mp.mpf(10) ** -36:
            break
        E = new
    E = -E if M < 0 else E
    den = 1 - e * mp.cos(E)
    return mp.cos(om) * ((mp.cos(E) - e) / den + e) - \
        mp.sin(om) * mp.sqrt((1 - e) * (1 + e)) * mp.sin(E) / den


@pytest.mark.parametrize("e", [0.0, 1e-300, 3e-6, 0.3, 0.5, 0.9, 0.99, 0.999])
@pytest.mark.parametrize("span,P", [(3000.0, 2.0), (3000.0, 1000.0), (1.0, 4e5), (2.0 ** 20, 1.0)])
def test_column(host, e, span, P):
    rng = np.random.default_rng(5)
    tsh = 62 - int(np.frexp(span)[1])
    m = ctypes.c_int64()
    for k in range(24):
        om, M0 = rng.uniform(-7, 7), rng.uniform(0, 2 * np.pi)
        t0 = int(rng.integers(-2 ** 62, 2 ** 61))
        t = int(rng.integers(0, 2 ** 62 - max(t0, 0)))
        if k % 3 == 0:                       # near pericentre: M of size 10^-9 .. 1
            M = 10.0 ** rng.uniform(-9, 0) * rng.choice([-1, 1])
            M0 = (2 * np.pi * (((t + t0) * 2.0 ** -tsh) / P) - M) % (2 * np.pi)
        if k == 1:
            om, M0 = 0.0, 0.0
        if k == 2:
            t, t0, M0 = 0, 0, np.pi
        assert host.column(tsh, t0, P, e, om, M0, t, ctypes.byref(m)) == 1
        dt = mpmath.mpf(t + t0) * mpmath.mpf(2) ** -tsh
        want = _exact(dt, P, e, om, M0)
        kap = 1.0 / (1.0 - e)
        tol = 2 * kap ** 2 * (2 * np.pi * (1 + 2 * span / P) * 2.0 ** -57 + 2.0 ** -53 * kap)
        assert abs(mpmath.mpf(m.value) / 2 ** 61 - want) <= tol


@pytest.mark.parametrize("P,e,om,M0", [(0.0, 0.1, 1, 1), (-3.0, 0.1, 1, 1), (np.nan, 0.1, 1, 1),
                                       (np.inf, 0.1, 1, 1), (5e-324, 0.1, 1, 1),
                                       (1e-7, 0.1, 1, 1), (3.0, -1e-9, 1, 1), (3.0, 1.0, 1, 1),
                                       (3.0, 0.9991, 1, 1), (3.0, np.nan, 1, 1),
                                       (3.0, 0.1, 1e4, 1), (3.0, 0.1, np.nan, 1),
                                       (3.0, 0.1, 1, np.inf), (3.0, 0.1, 1, -5000.0)])
def test_handed_over(host, P, e, om, M0):
    m = ctypes.c_int64()
    assert host.column(50, 0, P, e, om, M0, 12345, ctypes.byref(m)) == 0


def test_small_steps(host):
    rng = np.random.default_rng(6)
    one61, one62 = 1 << 61, 1 << 62
    for k in range(4000):
        den = int(2.0 ** rng.uniform(-9.9, 1) * one61) | int(rng.integers(1, 512))
        den = min(den, one62 - 1)
        num = int(rng.uniform(-1, 1) * den) if k % 3 else den * (1 if k % 2 else -1)
        q = host.quotient(num, den)
        assert abs(q * den - num * one61) <= 16 * den                 # 16 units of 2^-61
        y = max(1 << 40, one62 - 1 - k if k % 2 else int(rng.uniform(0.001, 1) * one62))
        y = max(y, int(0.001 * one62))
        # an FP32 correction of a root good to 2^-30
        assert abs(host.root(y) ** 2 - y * one62) <= 2 ** -51.0 * y * one62
        dn = int(rng.integers(one61, one62))
        assert abs(host.inverse(dn) * dn - (1 << 124)) <= 2 ** -57.0 * 2.0 ** 124


def test_powers_of_two(host):
    """2^(n + f): half an ulp of the rounding and the series' 2^-57."""
    mp = mpmath.mp
    mp.dps = 40
    rng = np.random.default_rng(7)
    one62 = 1 << 62
    for k in range(2000):
        f = [0, one62 - 1, (1 << 54) - 1, 1 << 54][k] if k < 4 else int(rng.integers(0, one62))
        n = int(rng.integers(-1000, 1000)) if k % 2 else 0
        got, want = mp.mpf(host.power(n, f)), mp.mpf(2) ** (n + mp.mpf(f) / one62)
        assert abs(got - want) <= mp.mpf(2) ** (n - 53) + want * mp.mpf(2) ** -57
    assert host.power(3, 0) == 8.0
