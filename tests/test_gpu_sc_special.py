"""The single-component boundary cells' kernel (csrc/sc_special.cuh: blocks of 32 listed cells)
and the collision's two halves against the C oracle, at lattice sizes around a block's 32 cells and
128 cells, with inflow, outflow, solid, adiabatic and free-slip cells.  FP64 on both sides; the
device's sums and factors differ from the oracle's by rounding: 1e-12 of each field's magnitude (the
bound of the reference's short runs), velocities against the largest velocity."""
import numpy as np
import pytest

import lbmgpu
from oracle import cases, sc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 7])
@pytest.mark.parametrize("freeslip_z", [False, True])
@pytest.mark.parametrize("shape", [(4, 3, 3), (8, 4, 4), (9, 5, 33), (31, 11, 4)])
def test_channel_matches_the_oracle(shape, freeslip_z, steps):
    cells, p = cases.channel_sc(*shape, freeslip_z=freeslip_z)
    with lbmgpu.Lattice(*cells.shape, p["nu"], p["R"], p["gamma"], p["prtl"]) as lat:
        lat.upload(cells)
        lat.init()
        lat.step(steps)
        assert lat.synchronize() == 0
        got = cells.copy()
        lat.download(got)
    want = cells.copy()
    o = sc.OracleSC(want, p["nu"], p["R"], p["gamma"], p["prtl"])
    o.init()
    o.loop(steps)
    fl = cells["type"] == cases.TYPE_F
    vs = max(np.abs(want[k][fl]).max() for k in "uvw")
    for k in ("rho", "temp", "p", "rhoe", "f", "g", "fpc", "gpc"):
        assert np.abs(got[k][fl] - want[k][fl]).max() <= 1e-12 * np.abs(want[k][fl]).max(), k
    for k in "uvw":
        assert np.abs(got[k][fl] - want[k][fl]).max() <= 1e-12 * vs, k
