"""lbmgpu_vtk_fields into page-locked memory: the values of a call with pageable memory, to the bit, where
the staging buffer holds the whole lattice and where it takes two pieces (104 B a cell of a nine-species
lattice, 256 MiB of staging)."""
import ctypes

import numpy as np
import pytest
import torch

import lbmgpu
import mech
import workloads as W

pytestmark = pytest.mark.gpu


def call(lat, out):
    out[:] = np.nan
    rc = lat.L.lbmgpu_vtk_fields(lat.h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), ctypes.c_size_t(out.size), 0)
    assert rc == 0
    return out


def both(lat, per_cell, ncell):
    n = (per_cell + 2) * ncell + 5
    pageable = call(lat, np.empty(n, np.float32))
    pinned = call(lat, torch.empty(n, dtype=torch.float32, pin_memory=True).numpy())
    assert np.isnan(pageable[-5:]).all() and not np.isnan(pageable[:-5]).any()
    assert np.array_equal(pageable, pinned, equal_nan=True)


@pytest.mark.parametrize("shape", [(3, 3, 3), (31, 15, 14), (57, 49, 41)])
def test_single_component(shape):
    cells, p = W.channel_sc(*shape)
    with lbmgpu.Lattice(*cells.shape, p["nu"], p["R"], p["gamma"], p["prtl"]) as lat:
        lat.upload(cells)
        lat.init()
        lat.step(2)
        both(lat, 7, cells.size)


@pytest.mark.parametrize("n", [4, 33])
def test_multicomponent(n):
    m = mech.h2_air_9()
    mix, sp = W.mixing_layer_mc(m, n)
    with lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS) as lat:
        lat.upload(mix, sp)
        lat.init()
        lat.step(1)
        both(lat, 8 + 2 * lat.ns, mix.size)


def test_two_pieces():
    m = mech.h2_air_9()
    mix, sp = W.mixing_layer_mc(m, 2, NY=194, NZ=194)  # its outermost and first interior planes, repeated
    nx = 68
    assert 104 * nx * mix[0].size > 256 << 20
    with lbmgpu.Lattice(nx, *mix.shape[1:], mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS,
                        precision=lbmgpu.FP32) as lat:
        for i in range(nx):
            q = 0 if i in (0, nx - 1) else 1
            lat.upload_planes(i, mix[q:q + 1], [a[q:q + 1] for a in sp])
        both(lat, 8 + 2 * lat.ns, nx * mix[0].size)
