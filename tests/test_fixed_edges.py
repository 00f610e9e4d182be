"""Edges of csrc/joker_fixed.cuh, compiled for the host."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "thejoker_gb300", "csrc")
SOURCE = r"""
#include "joker_fixed.cuh"
using namespace joker::fx;
extern "C" int64_t column(double P, double e, double om, double M0, uint64_t t) {
    Orbit o;
    return o.init(52, 0, P, e, om, M0) ? o.column(t) : INT64_MIN;
}
extern "C" int refused_then_bad(double P, double e) {
    alignas(Orbit) unsigned char mem[sizeof(Orbit)];
    std::memset(mem, 0xff, sizeof mem);              // NaNs
    Orbit *o = reinterpret_cast<Orbit *>(mem);
    return o->init(52, 0, P, e, 1.0, 1.0) ? -1 : (int)o->bad();
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("edges")
    src, so = str(d / "e.cc"), str(d / "e.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    CSRC, src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.column.argtypes = [ctypes.c_double] * 4 + [ctypes.c_uint64]
    lib.column.restype = ctypes.c_int64
    lib.refused_then_bad.argtypes = [ctypes.c_double] * 2
    return lib


@pytest.mark.parametrize("om,M0", [(1.0, 2.0), (-0.0, -0.0), (-3.0, 6.0)])
def test_negative_zero(host, om, M0):
    """An eccentricity of -0 is 0."""
    for t in (0, 12345 << 30, 1 << 61):
        assert host.column(30.0, -0.0, om, M0, t) == host.column(30.0, 0.0, om, M0, t)


@pytest.mark.parametrize("P,e", [(0.0, 0.1), (30.0, 2.0), (float("nan"), 0.1)])
def test_refused_orbit_is_not_bad(host, P, e):
    """bad() is stored for every sample: defined for one that init refused."""
    assert host.refused_then_bad(P, e) == 0
