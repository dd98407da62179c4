"""The device's population update (csrc/mc_relax.cuh) against the host build of the per-cell functions
it restates, on small ragged periodic boxes: a block's last threads past the lattice, ghost cells
between the cells of a warp, vanishing species (they keep their populations, along the directions
where chemistry adds nothing) and the first step's in-place populations.  FP64 sides differ by the
rounding of regrouped sums and by exp and log: 1e-12 of each field's scale after a few steps, 1e-10
for the heat release.  FP32 storage: a flipped last bit of a stored population, 6e-8 of the plane's
spread, held to 1e-6."""
import numpy as np
import pytest

import lbmgpu
import mech
import workloads as W
from mc_common import SP0, build_host_lib, host_run, rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hostlib(tmp_path_factory):
    return build_host_lib(tmp_path_factory.mktemp("host"), contract=False)


@pytest.mark.parametrize("steps", [1, 3])
@pytest.mark.parametrize("chem", [lbmgpu.CHEM_OFF, lbmgpu.CHEM_REF_EXPLICIT])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("name,shape", [("h2_air_9", (8, 3, 5)), ("h2_air_9", (9, 4, 31)), ("ch4_2s", (11, 6, 2)),
                                        ("ch4_2s", (8, 8, 8))])
def test_update_matches_the_host_cells(hostlib, name, shape, precision, chem, steps):
    m = getattr(mech, name)()
    fuel = dict(fuel="H2", Y_H2=0.03) if name == "h2_air_9" else dict(fuel="CH4", Y_H2=0.05)
    mix, sp = W.mixing_layer_mc(m, shape[0], NY=shape[1], NZ=shape[2], T_hi=1600.0, **fuel)
    want, st = host_run(hostlib, m, mix, sp, chem, steps, precision=precision)[:2]
    with lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS, chem=chem,
                        precision=lbmgpu.FP64 if precision == "fp64" else lbmgpu.FP32,
                        library=lbmgpu.NOFMA_LIB_PATH) as lat:
        lat.upload(mix, sp)
        lat.init()
        lat.step(steps)
        assert lat.synchronize() == st
        got, gsp = mix.copy(), [a.copy() for a in sp]
        lat.download(got, gsp)
    fl = (mix["type"] == W.TYPE_F).reshape(-1)
    tol, tol_hrr = (1e-12, 1e-10) if precision == "fp64" else (1e-6, 1e-5)
    for q, k in ((0, "rho"), (4, "temp"), (5, "p"), (6, "rhoe")):
        assert rel(got[k].reshape(-1)[fl], want[q][fl]) < tol, k
    for a in range(len(sp)):
        assert rel(gsp[a]["rho"].reshape(-1)[fl], want[SP0 + 8 * a][fl]) < tol, a
    if chem:
        assert rel(got["HRR"].reshape(-1)[fl], want[13][fl]) < tol_hrr
