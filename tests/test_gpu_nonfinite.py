"""A state that is no longer finite spreads as in the reference: one cell starts at a temperature or
pressure that is not a number (or is infinite), and after a few steps the same values of the same cells
are finite as in the C oracle (single component) and in the host build of the per-cell functions
(multicomponent), which form every product of a sum, the ones with zero included."""
import numpy as np
import pytest

import lbmgpu
import mech
import workloads as W
from mc_common import SP0, build_host_lib, host_run
from oracle import cases, sc

pytestmark = pytest.mark.gpu

BAD = [("temp", np.nan), ("p", np.nan), ("temp", np.inf), ("p", -np.inf)]


def same(got, want, name):
    assert np.array_equal(np.isfinite(got), np.isfinite(want)), name


@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("field,value", BAD)
@pytest.mark.parametrize("walls", [False, True])
def test_single_component(walls, field, value, steps):
    cells, p = cases.channel_sc(11, 8, 7) if walls else cases.tgv_sc(9, Re=10.0)
    cells[field][4, 4, 4] = value
    with lbmgpu.Lattice(*cells.shape, p["nu"], p["R"], p["gamma"], p["prtl"]) as lat:
        lat.upload(cells)
        lat.init()
        lat.step(steps)
        assert lat.synchronize() & 1
        got = cells.copy()
        lat.download(got)
    want = cells.copy()
    with np.errstate(all="ignore"):
        o = sc.OracleSC(want, p["nu"], p["R"], p["gamma"], p["prtl"])
        o.init()
        o.loop(steps)
    fl = cells["type"] == cases.TYPE_F
    assert not np.isfinite(want["g"][fl]).all() and np.isfinite(want["g"][fl]).any()
    for k in ("rho", "u", "v", "w", "temp", "p", "rhoe", "f", "g"):
        same(got[k][fl], want[k][fl], k)


@pytest.fixture(scope="module")
def hostlib(tmp_path_factory):
    return build_host_lib(tmp_path_factory.mktemp("host"), contract=False)


@pytest.mark.parametrize("steps", [1, 2, 3])
@pytest.mark.parametrize("field,value", BAD[:2])
@pytest.mark.parametrize("name,walls,chem", [("h2_air_9", False, 0), ("h2_air_9", True, 0), ("h2_air_9", False, 1),
                                             ("ch4_2s", False, 1), ("c3h8_2s", False, 1)])
def test_multicomponent(hostlib, name, walls, chem, field, value, steps):
    m = getattr(mech, name)()
    fuel = {"h2_air_9": "H2", "ch4_2s": "CH4", "c3h8_2s": "C3H8"}[name]
    mix, sp = W.flame_channel_mc(m, 11, 8, 7) if walls else W.mixing_layer_mc(m, 9, T_hi=1500.0, fuel=fuel)
    mix[field][4, 4, 4] = value
    fl = (mix["type"] == W.TYPE_F).reshape(-1)
    want, st, pops = host_run(hostlib, m, mix, sp, chem, steps, pops=True)
    with lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS, chem=chem,
                        library=lbmgpu.NOFMA_LIB_PATH) as lat:
        lat.upload(mix, sp)
        lat.init()
        lat.step(steps)
        assert lat.synchronize() == st
        got, gsp = mix.copy(), [a.copy() for a in sp]
        lat.download(got, gsp)
    for q, k in ((0, "rho"), (1, "u"), (2, "v"), (3, "w"), (4, "temp"), (5, "p"), (6, "rhoe")):
        same(got[k].reshape(-1)[fl], want[q][fl], k)
    g = pops[27 * len(sp):]
    assert not np.isfinite(g[:, fl]).all() and np.isfinite(g[:, fl]).any()
    same(got["g"].reshape(-1, 27)[fl].T, g[:, fl], "g")
    for a in range(len(sp)):
        same(gsp[a]["f"].reshape(-1, 27)[fl].T, pops[27 * a:27 * (a + 1)][:, fl], ("f", a))
        same(gsp[a]["rho"].reshape(-1)[fl], want[SP0 + 8 * a][fl], ("rho", a))
        same(gsp[a]["X"].reshape(-1)[fl], want[SP0 + 8 * a + 4][fl], ("X", a))
