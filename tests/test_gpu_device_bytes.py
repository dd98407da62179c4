"""lbmgpu_device_bytes counts what the handle holds: an evaluation's and an augmentation's buffers
go when the call ends, a grown sample set replaces the old one, and an upload with other boundary
cells replaces the boundary store."""
import numpy as np
import pytest

import lbmgpu
from oracle import cases
from test_gpu_surrogate import lattice

pytestmark = pytest.mark.gpu

ROW = (lbmgpu.SUR_IN + lbmgpu.SUR_OUT) * 4 + 1  # a sample row: features, targets, whether it is valid


def test_surrogate_calls():
    x = np.random.default_rng(1).standard_normal((500, 12), dtype=np.float32)
    lat, m, mix, sp = lattice()
    with lat:
        lat.upload(mix, sp)
        lat.init()
        lat.surrogate_collect(True, stride=1, capacity=2000)
        lat.step(2)
        lat.surrogate_collect(False)
        before = lat.device_bytes()
        lat.surrogate_eval(x)
        assert lat.device_bytes() == before
        n = lat.surrogate_stats()["samples"]
        lat.surrogate_augment(2500 - n, seed=1)  # grows the set to 2,500 rows
        assert lat.device_bytes() == before + 500 * ROW
        lat.surrogate_load_samples(np.zeros((4000, 12), np.float32), np.zeros((4000, 10), np.float32))
        assert lat.device_bytes() == before + 2000 * ROW
        with pytest.raises(lbmgpu.LbmGpuError):
            lat.surrogate_collect(True, capacity=1 << 42)
        assert lat.device_bytes() == before + 2000 * ROW


def test_boundary_store():
    walled, p = cases.channel_sc(8, 5, 4)
    periodic = walled.copy()
    periodic["type"][1:-1, 1:-1, 1:-1] = cases.TYPE_F
    for f in (0, -1):
        periodic["type"][f] = periodic["type"][:, f] = periodic["type"][:, :, f] = cases.TYPE_P
    with lbmgpu.Lattice(*walled.shape, p["nu"], p["R"], p["gamma"], p["prtl"]) as lat:
        lat.upload(periodic)
        before = lat.device_bytes()
        lat.upload(walled)
        assert lat.device_bytes() > before
        lat.upload(periodic)
        assert lat.device_bytes() == before
