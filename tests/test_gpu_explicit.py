"""The explicit chemistry's two kinetics on the device: the compiled H2/air mechanism
(kinetics_h2_air_9.cuh, net_t) against the dense tables (gas::net_production_dense), which a
mechanism with one rate constant an ulp off runs.  The two evaluate the same rate laws in another
order of products, so a few steps of the hot slab agree to rounding: each step adds a relative 1e-14
of the rates (their order of 10 products and an exponential of an argument near 100) to increments
below the fields, held here to 1e-12 of each field's scale, the heat release to 1e-10."""
import numpy as np
import pytest

import lbmgpu
import mech
import workloads as W
from mc_common import rel

pytestmark = pytest.mark.gpu


def run(m, mix, sp, precision, steps):
    with lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS,
                        chem=lbmgpu.CHEM_REF_EXPLICIT, precision=precision) as lat:
        lat.upload(mix, sp)
        lat.init()
        lat.step(steps)
        assert lat.synchronize() == 0
        c, s = mix.copy(), [a.copy() for a in sp]
        lat.download(c, s)
    return c, s


@pytest.mark.parametrize("shape", [(6, 5, 4), (11, 8, 3), (16, 16, 16)])
@pytest.mark.parametrize("precision", [lbmgpu.FP64, lbmgpu.FP32])
def test_compiled_and_dense_rates_agree(precision, shape):
    m = mech.h2_air_9()
    mix, sp = W.mixing_layer_mc(m, shape[0], NY=shape[1], NZ=shape[2], T_hi=1800.0)
    other = mech.h2_air_9()
    other.A[2] = np.nextafter(other.A[2], np.inf)
    a, sa = run(m, mix, sp, precision, 5)
    b, sb = run(other, mix, sp, precision, 5)
    fl = mix["type"] == W.TYPE_F
    # FP32 storage: a flipped last bit of a stored population is 6e-8 of its plane's spread
    tol, tol_hrr = (1e-12, 1e-10) if precision == lbmgpu.FP64 else (1e-6, 1e-5)
    for k in ("rho", "temp", "p", "rhoe"):
        assert rel(a[k][fl], b[k][fl]) < tol, k
    for x, y in zip(sa, sb):
        assert rel(x["rho"][fl], y["rho"][fl], np.abs(b["rho"][fl]).max()) < tol
    assert np.abs(b["HRR"][fl]).max() > 0
    assert rel(a["HRR"][fl], b["HRR"][fl]) < tol_hrr
