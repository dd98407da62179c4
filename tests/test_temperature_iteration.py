"""The moments' temperature iteration (gas::T_from_u_tab, csrc/gas.cuh): where its last steps cross a
polynomial range's end the result is as exact as elsewhere.  The mechanism's c_p is raised by a tenth
above T_mid, h left continuous, so that a step of 1e-8 T across T_mid is off by a tenth of itself; the
iteration starts such steps away from the solution.  Bound: nine terms of some 20 roundings each,
2e-14 of a u that is of the order of c_v T; held to 1e-13."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import mech
from mc_common import CSRC, ROOT

D = ctypes.c_double


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host") / "libthermo.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(ROOT, "tests", "host", "thermo_host.cpp"), "-o", out], check=True)
    L = ctypes.CDLL(out)
    L.energy.restype = D
    return L


def kinked(name):
    m = getattr(mech, name)()
    for k in range(m.n_species):
        Tm = m.T_mid[k] = 1000.0
        lo, hi = m.nasa_lo[k], m.nasa_hi[k]
        for i in range(7):
            hi[i] = lo[i]
        hi[0] = lo[0] * 1.1
        hi[5] = lo[5] - 0.1 * lo[0] * Tm  # h continuous at T_mid
    return m


@pytest.mark.parametrize("fast", [0, 1])
@pytest.mark.parametrize("name", ["h2_air_9", "ch4_2s"])
def test_steps_across_a_range_end(lib, name, fast):
    m = kinked(name)
    n = m.n_species
    Y = np.random.default_rng(1).uniform(0.1, 1.0, n)
    Y /= Y.sum()
    Yp = Y.ctypes.data_as(ctypes.POINTER(D))
    for side in (-1.0, 1.0):
        for d in (1e-6, 9e-9, 5e-9, 1e-9, 1e-10):
            T_true = 1000.0 * (1.0 + side * d / 2)
            u = lib.energy(ctypes.byref(m), Yp, D(T_true))
            T = D()
            it = lib.temperature(ctypes.byref(m), fast, Yp, D(u), D(T_true * (1.0 - side * d)), ctypes.byref(T))
            assert it > 0
            assert abs(T.value - T_true) < 1e-13 * T_true, (side, d)


@pytest.mark.parametrize("fast", [0, 1])
def test_far_starts(lib, fast):
    m = mech.h2_air_9()
    rng = np.random.default_rng(2)
    for _ in range(50):
        Y = rng.uniform(0.0, 1.0, 9)
        Y /= Y.sum()
        Yp = Y.ctypes.data_as(ctypes.POINTER(D))
        T_true = rng.uniform(250.0, 3000.0)
        if abs(T_true - 1000.0) < 1.0:
            continue
        u = lib.energy(ctypes.byref(m), Yp, D(T_true))
        T = D()
        assert 0 < lib.temperature(ctypes.byref(m), fast, Yp, D(u), D(rng.uniform(250.0, 3000.0)), ctypes.byref(T)) < 30
        assert abs(T.value - T_true) < 1e-13 * T_true
