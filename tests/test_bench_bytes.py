"""The byte counts behind the bench's hbm_gbs_step: planes that each kernel of a step loads and stores
(csrc/mc_moments.cuh, mc_eflux.cuh, and mc_props_cell, mc_chem_state, mc_chem_explicit of mc_cell.cuh),
nine species."""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

import bench  # noqa: E402

PLANES = {
    "k_mc_gather": 47,      # written: rho, u, P, rhoE; rho_a, j_a
    "k_mc_diffuse": 109,    # read 82 (p, X_a, rho_a, j_a, 36 D_ab), written 27
    "k_mc_thermo": 83,      # read 42 (rho, u, rhoE, T; rho_a, u_a; no P tensor), written 41
    "k_mc_props": 126,      # read 49 (no mixture velocity, no P tensor), written 77
    "k_mc_eflux": 57,       # read 54, written 3
    "k_mc_chem": 21,        # read 11, written 10
    "k_mc_explicit": 49,    # read 39, written 10
}


@pytest.mark.parametrize("pop_bytes", [4, 8])
@pytest.mark.parametrize("reaction", [False, True])
def test_step_bytes(reaction, pop_bytes):
    for kernel, planes in PLANES.items():
        pops = 270 * pop_bytes if kernel == "k_mc_gather" else 0
        assert bench.step_bytes(kernel, pop_bytes, reaction) == pops + 8 * planes, kernel
    assert bench.step_bytes("k_mc_relax", pop_bytes, reaction) == bench.mc_bytes("k_mc_relax", pop_bytes, reaction)
