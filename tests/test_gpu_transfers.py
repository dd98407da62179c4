"""Record transfers and output fields in several chunks (the host copies one while the device packs the
next): lattices of 1 to 5 chunks of 8,192 cells, with a short last one.  Copies only, so every value is
exact: records uploaded and read back, a stepped state through a second lattice, and the fields against
the records rounded to single precision."""
import ctypes

import numpy as np
import pytest

import lbmgpu
import mech
import workloads as W

pytestmark = pytest.mark.gpu


def fields(lat, per_cell, ncell):
    out = np.full((per_cell + 2) * ncell, np.nan, np.float32)
    rc = lat.L.lbmgpu_vtk_fields(lat.h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), ctypes.c_size_t(out.size), 0)
    assert rc == 0
    return out


def planes(out, shape, first, width=1):
    n = int(np.prod(shape))
    a = out[first * n:(first + width) * n]
    return a.reshape(shape[::-1] + ((width,) if width > 1 else ())).transpose((2, 1, 0) + ((3,) if width > 1 else ()))


@pytest.mark.parametrize("shape", [(6, 5, 4), (31, 15, 14), (41, 37, 19)])
def test_single_component(shape):
    cells, p = W.channel_sc(*shape)
    args = (p["nu"], p["R"], p["gamma"], p["prtl"])
    with lbmgpu.Lattice(*cells.shape, *args) as lat:
        lat.upload(cells)
        lat.init()
        lat.step(3)
        got = cells.copy()
        lat.download(got)
        out = fields(lat, 7, cells.size)
    for k, name in ((0, "rho"), (5, "temp"), (6, "p")):
        assert np.array_equal(planes(out, cells.shape, k), got[name].astype(np.float32)), name
    vel = planes(out, cells.shape, 1, 3)
    for d, name in enumerate("uvw"):
        assert np.array_equal(vel[..., d], got[name].astype(np.float32)), name
    assert np.array_equal(planes(out, cells.shape, 4), cells["type"].astype(np.float32))
    # the stepped records through another lattice: the fluid cells' state comes back to the bit
    with lbmgpu.Lattice(*cells.shape, *args) as lat:
        lat.upload(got)
        back = got.copy()
        lat.download(back)
    fluid = cells["type"] == 0
    for name in ("f", "g", "rho", "u", "v", "w", "temp", "p"):
        assert np.array_equal(back[name][fluid], got[name][fluid]), name


@pytest.mark.parametrize("n", [6, 24, 32])
def test_multicomponent(n):
    m = mech.h2_air_9()
    mix, sp = W.mixing_layer_mc(m, n)
    kw = dict(mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS)
    with lbmgpu.Lattice(*mix.shape, **kw) as lat:
        lat.upload(mix, sp)
        lat.init()
        lat.step(2)
        got, gsp = mix.copy(), [s.copy() for s in sp]
        lat.download(got, gsp)
        out = fields(lat, 8 + 2 * lat.ns, mix.size)
    inner = (slice(1, -1),) * 3
    for k, name in ((0, "rho"), (5, "temp"), (6, "p"), (7, "HRR")):
        assert np.array_equal(planes(out, mix.shape, k)[inner], got[name].astype(np.float32)[inner]), name
    for a, s in enumerate(gsp):
        assert np.array_equal(planes(out, mix.shape, 8 + a)[inner], s["X"].astype(np.float32)[inner]), a
    with lbmgpu.Lattice(*mix.shape, **kw) as lat:
        lat.upload(got, gsp)
        back, bsp = got.copy(), [s.copy() for s in gsp]
        lat.download(back, bsp)
    for name in ("g", "rho", "temp", "p"):
        assert np.array_equal(back[name][inner], got[name][inner]), name
    for s, b in zip(gsp, bsp):
        assert np.array_equal(b["f"][inner], s["f"][inner])
