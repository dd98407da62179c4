"""Steps captured into a CUDA graph on the handle's stream (lbmgpu_get_stream): the fork to the side
stream and its join, and the launches that start while the kernel before drains, are captured; two steps
replayed are two steps, to the bit."""
import numpy as np
import pytest
import torch

import lbmgpu
import mech
import workloads as W

pytestmark = pytest.mark.gpu


def check(make, state):
    out = []
    for graphed in (False, True):
        with make() as lat:
            lat.upload(*state)
            lat.init()
            lat.step(2)  # the buffers are back where they were after an even number of steps
            lat.synchronize()
            if graphed:
                stream = torch.cuda.ExternalStream(lat.stream())
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
                    lat.step(2)
                with torch.cuda.stream(stream):
                    for _ in range(3):
                        graph.replay()
                lat.synchronize()
                del graph
            else:
                lat.step(6)
            assert lat.synchronize() == 0
            got = [state[0].copy()] + [[a.copy() for a in s] for s in state[1:]]
            lat.download(*got)
            out.append([got[0]] + [a for s in got[1:] for a in s])
    for a, b in zip(*out):
        for name in a.dtype.names:
            assert a[name].tobytes() == b[name].tobytes(), name


@pytest.mark.parametrize("walls", [False, True])
def test_single_component(walls):
    cells, p = W.channel_sc(31, 13, 9) if walls else W.tgv_sc(17, Re=10.0)
    check(lambda: lbmgpu.Lattice(*cells.shape, p["nu"], p["R"], p["gamma"], p["prtl"]), (cells,))


@pytest.mark.parametrize("chem", [lbmgpu.CHEM_OFF, lbmgpu.CHEM_REF_EXPLICIT, lbmgpu.CHEM_ROSENBROCK])
@pytest.mark.parametrize("walls", [False, True])
def test_multicomponent(walls, chem):
    m = mech.h2_air_9()
    mix, sp = W.flame_channel_mc(m, 24, 6, 5) if walls else W.mixing_layer_mc(m, 13, NY=9, NZ=7, T_hi=1800.0)
    check(lambda: lbmgpu.Lattice(*mix.shape, mech=m, dtype=W.MIXTURE_MC, species_dtype=W.SPECIES, dx_dt=W.FLAME_UNITS,
                                 chem=chem), (mix, sp))
