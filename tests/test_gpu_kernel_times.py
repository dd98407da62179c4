"""lbmgpu_kernel_times: launches per kind and step, one of the collision parameters' kernel in every
chemistry mode, and single-component times that do not overlap (their sum is within the steps' own
time)."""
import pytest

import lbmgpu
import mech
import workloads as W

pytestmark = pytest.mark.gpu

STEPS = 4


def counts(lat, steps=STEPS):
    lat.step(2)
    lat.profile(True)
    elapsed = lat.time_steps(steps)
    launches, ms = lat.kernel_times()
    lat.profile(False)
    return launches, ms, elapsed


@pytest.mark.parametrize("precision", [lbmgpu.FP64, lbmgpu.FP32])
@pytest.mark.parametrize("chem", [lbmgpu.CHEM_OFF, lbmgpu.CHEM_REF_EXPLICIT, lbmgpu.CHEM_ROSENBROCK])
@pytest.mark.parametrize("walls", [False, True])
def test_multicomponent(walls, chem, precision):
    m = mech.h2_air_9()
    mix, sp = W.flame_channel_mc(m, 16, 4, 4) if walls else W.mixing_layer_mc(m, 6)
    with lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS, chem=chem,
                        precision=precision) as lat:
        lat.upload(mix, sp)
        lat.init()
        launches, ms, _ = counts(lat)
    per_step = [1, 1, int(walls), 1, 0, 2, 1, int(chem != lbmgpu.CHEM_OFF)]
    assert launches == [STEPS * k for k in per_step]
    assert all((t > 0) == (k > 0) for t, k in zip(ms, per_step))


@pytest.mark.parametrize("walls", [False, True])
def test_single_component(walls):
    cells, p = W.channel_sc(97, 41, 30) if walls else W.tgv_sc(24, Re=10.0)
    with lbmgpu.Lattice(*cells.shape, p["nu"], p["R"], p["gamma"], p["prtl"]) as lat:
        lat.upload(cells)
        lat.init()
        launches, ms, elapsed = counts(lat, 20)
    assert launches == [20, 20, 20 * int(walls), 0, 0, 0, 0, 0]
    assert sum(ms) <= elapsed
