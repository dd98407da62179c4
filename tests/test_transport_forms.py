"""The two FP64 forms of the collision parameters (csrc/mc_cell.cuh, mc_transport_f64): the reference's
quotients, which the host build's steps and the comparisons with the reference run, against the
device's square roots, reciprocals and shared pair coefficients.  Over temperatures, pressures,
compositions (traces at the reference's floor among them) and species velocities: the same
diffusion coefficients to the bit, and every other plane within 1e-12 -- sums of nine positive terms
of some ten roundings each; the force against the cell's largest, its terms being of either sign."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import mech
import workloads as W
from mc_common import CSRC, ROOT, SP0, nrec

N = 4000


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host") / "libprops.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(ROOT, "tests", "host", "props_host.cpp"), "-o", out], check=True)
    return ctypes.CDLL(out)


def states(m, seed):
    """Record planes of N cells: rho, u, T, p, rhoE, and per species rho_a, u_a, X_a."""
    ns = m.n_species
    rng = np.random.default_rng(seed)
    R = np.zeros((nrec(ns), N))
    Wk = np.array([m.W[k] for k in range(ns)])
    X = rng.uniform(0, 1, (ns, N)) ** 4 * (rng.uniform(0, 1, (ns, N)) < 0.7) + 1e-8
    X /= X.sum(0)
    T = rng.uniform(250, 3000, N)
    Y = X * Wk[:, None] / (X * Wk[:, None]).sum(0)
    R[0] = rng.uniform(0.2, 3.0, N)
    R[4] = T * W.t_lattice(1.0)
    R[5] = W.p_lattice(101325.0) * np.exp(rng.uniform(-2, 2, N))
    R[6] = R[0] * 0.1
    for d in range(3):
        R[1 + d] = rng.normal(0, 1e-2, N)
    for a in range(ns):
        R[SP0 + 8 * a] = R[0] * Y[a]
        for d in range(3):
            R[SP0 + 8 * a + 1 + d] = R[1 + d] + rng.normal(0, 1e-3, N)
        R[SP0 + 8 * a + 4] = X[a]
    return R


@pytest.mark.parametrize("name", ["h2_air_9", "ch4_2s", "c3h8_2s"])
def test_forms_agree(lib, name):
    m = getattr(mech, name)()
    ns = m.n_species
    R = states(m, 5)
    planes = 5 * ns + 8 + ns * (ns - 1) // 2
    out = np.zeros((2, planes, N))
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    for k in range(2):
        got = lib.collision_params(ctypes.byref(m), ctypes.c_float(W.FLAME_UNITS[0]), ctypes.c_float(W.FLAME_UNITS[1]),
                                   ctypes.c_long(N), P(R), 1 - k, P(out[k]))
        assert got == planes
    exact, device = out
    assert np.isfinite(exact).all()
    om = np.r_[0:ns, 5 * ns:5 * ns + 4, planes - 1]  # om_a, omega, omega_1, theta, U, R/W
    assert (exact[om] != 0).all()
    assert np.abs(device[om] / exact[om] - 1).max() < 1e-12
    D = slice(5 * ns + 7, planes - 1)
    assert (exact[D] > 0).all() and np.array_equal(exact[D], device[D])
    rho_a = np.array([R[SP0 + 8 * a] for a in range(ns)])
    F = [(o[ns:4 * ns].reshape(ns, 3, N) * rho_a[:, None]) for o in out]
    scale = np.abs(F[0]).max((0, 1))
    assert (scale > 0).all()
    assert (np.abs(F[1] - F[0]).max((0, 1)) < 1e-12 * scale).all()
    assert not np.array_equal(exact, device)  # two forms, not one
