"""A step's kernels overlap: the chemistry beside the transport, the boundary cells beside the interior,
each kernel launched while the one before drains.  While kernels are timed they run one after the other
(lbmgpu_profile), so a timed run of the same steps has to give the same bits."""
import numpy as np
import pytest

import lbmgpu
import mech
import workloads as W

pytestmark = pytest.mark.gpu

STEPS = 12


def phases(lat):
    if lat.ns:
        lat.collide_species()
    lat.collide()
    lat.streaming()
    lat.tms_bc()
    lat.calculate_moment()


def run(make, state, timed, by_phase):
    with make() as lat:  # its own handle: FP32 storage rounds an upload against the shift before
        lat.upload(*state)
        lat.init()
        lat.profile(timed)
        if by_phase:
            for _ in range(STEPS):
                phases(lat)
        else:
            lat.step(STEPS)
        status = lat.synchronize()
        lat.profile(False)
        out = [state[0].copy()] + [[a.copy() for a in s] for s in state[1:]]
        lat.download(*out)
    return status, [out[0]] + [a for s in out[1:] for a in s]


def same(make, state):
    want = run(make, state, True, False)
    for by_phase in (False, True):
        got = run(make, state, False, by_phase)
        assert got[0] == want[0]
        for a, b in zip(got[1], want[1]):
            for name in a.dtype.names:
                assert a[name].tobytes() == b[name].tobytes(), name


@pytest.mark.parametrize("walls", [False, True])
def test_single_component(walls):
    cells, p = W.channel_sc(31, 13, 9) if walls else W.tgv_sc(17, Re=10.0)
    same(lambda: lbmgpu.Lattice(*cells.shape, p["nu"], p["R"], p["gamma"], p["prtl"]), (cells,))


@pytest.mark.parametrize("precision", [lbmgpu.FP64, lbmgpu.FP32])
@pytest.mark.parametrize("chem", [lbmgpu.CHEM_OFF, lbmgpu.CHEM_REF_EXPLICIT, lbmgpu.CHEM_ROSENBROCK])
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("name", ["h2_air_9", "ch4_2s"])
def test_multicomponent(name, walls, chem, precision):
    m = getattr(mech, name)()
    if name == "ch4_2s":
        if walls:
            pytest.skip("the walled layer is a 9-species case")
        mix, sp = W.mixing_layer_mc(m, 13, NY=9, NZ=7, T_hi=1800.0, fuel="CH4", Y_H2=0.05)
    else:
        mix, sp = W.flame_channel_mc(m, 24, 6, 5) if walls else W.mixing_layer_mc(m, 13, NY=9, NZ=7, T_hi=1800.0)
    same(lambda: lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS,
                                chem=chem, precision=precision), (mix, sp))


@pytest.mark.parametrize("walls", [False, True])
def test_surrogate_in_use(walls):
    m = mech.h2_air_9()
    mix, sp = W.flame_channel_mc(m, 24, 6, 5) if walls else W.mixing_layer_mc(m, 13, NY=9, NZ=7, T_hi=1800.0)

    def make():
        return lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS,
                              chem=lbmgpu.CHEM_ROSENBROCK, precision=lbmgpu.FP32)

    with make() as lat:
        lat.upload(mix, sp)
        lat.init()
        lat.surrogate_collect(True, stride=1, capacity=4 * mix.size)
        lat.step(4)
        lat.surrogate_collect(False)
        lat.surrogate_train(epochs=20, batch=256, lr=2e-3, seed=1)
        params = lat.surrogate_params()

    def with_surrogate():
        lat = make()
        lat.surrogate_params(params)
        lat.surrogate_enable(True, audit_period=100)
        return lat

    same(with_surrogate, (mix, sp))
    with with_surrogate() as lat:
        lat.upload(mix, sp)
        lat.init()
        lat.step(STEPS)
        lat.synchronize()
        st = lat.surrogate_stats()
    assert st["cells_predicted"] > 0 and st["cells_integrated"] + st["cells_audited"] > 0
