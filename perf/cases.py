"""What a user of this library has it do, as cases that can be timed and compared.

A pass is what the reference's driver loop does between two outputs: a number of time steps
through ``Lattice.step`` and then the output itself.  The output is either the cell records of
the whole lattice (``Lattice.download``: populations, post-collision populations and moments in
FP64, what a restart file holds) or the output fields (``lbmgpu_vtk_fields``: every cell array of
the reference's VTK file, FP32).  Cases that start over in each pass upload their set-up records
and initialise them first, as a program starts a run: they are the ones whose flow does not
stay stable over the thousands of steps that a state would otherwise take while it is timed.

The surrogate's case trains the chemistry network for an epoch and evaluates it.

Sizes are interior cells per axis (the ghost layer comes on top).
"""
import ctypes
import importlib
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "lattice-boltzmann-method_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
lbmgpu = importlib.import_module("lbmgpu")
mech = importlib.import_module("mech")
workloads = importlib.import_module("workloads")

_MECHS = {"h2_air_9": mech.h2_air_9, "ch4_2s": mech.ch4_2s, "c3h8_2s": mech.c3h8_2s}
_FUEL = {"h2_air_9": ("H2", 0.03), "ch4_2s": ("CH4", 0.05), "c3h8_2s": ("C3H8", 0.05)}
_CHEM = {"off": lbmgpu.CHEM_OFF, "explicit": lbmgpu.CHEM_REF_EXPLICIT, "ros2": lbmgpu.CHEM_ROSENBROCK}


def _sc(flow, nx, ny, nz, steps, out, **more):
    return dict(flow=flow, nx=nx, ny=ny, nz=nz, steps=steps, out=out, **more)


def _mc(flow, nx, ny, nz, steps, out, mechanism="h2_air_9", chem="off", precision="fp64", restart=False):
    return dict(flow=flow, nx=nx, ny=ny, nz=nz, steps=steps, out=out, mechanism=mechanism, chem=chem,
                precision=precision, restart=restart)


def listed():
    return [
        # a unit-test-sized box: launches and their gaps are all there is to it
        dict(_sc("tgv", 16, 16, 16, 200, "records", re=10.0), name="sc_tgv_16"),
        # the single-component headline: 64^3 Taylor-Green vortex, 1000 steps, state compared afterwards
        dict(_sc("tgv", 64, 64, 64, 1000, "records", re=400.0), name="sc_tgv_64"),
        # a production-sized single-component box with odd sides, between two field outputs
        dict(_sc("tgv", 150, 121, 113, 200, "fields", re=400.0), name="sc_tgv_150x121x113"),
        # inflow, outflow, wall and adiabatic boundaries around a channel flow
        dict(_sc("channel", 97, 41, 30, 500, "records"), name="sc_channel_97x41x30"),
        # the reacting fixture: 9 species, the reference's explicit chemistry, FP64, a handful of cells
        dict(_mc("slab", 8, 8, 8, 100, "records", chem="explicit"), name="mc_react_8"),
        # the 6-species methane mechanism, reacting, the FP64 reference mode
        dict(_mc("slab", 32, 32, 32, 100, "records", mechanism="ch4_2s", chem="explicit"), name="mc_ch4_32"),
        # non-reacting H2/air mixing in the FP64 reference mode, odd sides
        dict(_mc("slab", 48, 40, 37, 100, "records"), name="mc_mix_48x40x37"),
        # the mixing layer between characteristic inflow and outflow, FP64, from its start
        dict(_mc("inflow", 64, 48, 40, 100, "fields", restart=True), name="mc_inflow_64x48x40"),
        # the premixed flame channel: walls, characteristic outlets, explicit chemistry, FP32 storage
        dict(_mc("flame", 512, 8, 8, 200, "fields", chem="explicit", precision="fp32", restart=True),
             name="mc_flame_512x8x8"),
        # the decaying turbulent reacting layer with stiff chemistry, FP32 storage, from its start
        dict(_mc("turbulence", 64, 64, 64, 60, "fields", chem="ros2", precision="fp32", restart=True),
             name="mc_turb_64"),
        # a large periodic reacting slab with stiff chemistry, FP32 storage, between two field outputs
        dict(_mc("slab", 96, 96, 96, 40, "fields", chem="ros2", precision="fp32"), name="mc_react_96"),
        # the chemistry surrogate: one training epoch (forward and backward) and an evaluation
        dict(flow="surrogate", rows=200000, batch=4096, name="surrogate_200k"),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _steps(cells, budget, most):
    """Steps between two outputs: as many as keep a pass within `budget` cell updates."""
    return max(10, min(most, int(budget / cells)))


def draw(rng):
    flow = rng.choice(["tgv", "channel", "slab", "slab", "slab", "inflow", "flame", "turbulence", "surrogate"])
    if flow == "tgv":
        nx = _side(rng, 12, 150)
        ny, nz = (max(12, int(nx * rng.uniform(0.6, 1.1))) for _ in range(2))
        cells = nx * ny * nz
        return _sc("tgv", nx, ny, nz, _steps(cells, 1.5e8, 500), "records" if cells < 4e5 else "fields",
                   re=10.0 if min(nx, ny, nz) < 33 else 100.0)
    if flow == "channel":
        return _sc("channel", _side(rng, 16, 110), _side(rng, 8, 45), _side(rng, 8, 36), rng.randint(50, 400), "records")
    if flow == "slab":
        mechanism = rng.choice(["h2_air_9", "h2_air_9", "ch4_2s", "c3h8_2s"])
        precision = rng.choice(["fp64", "fp32"])
        chem = rng.choice(["off", "explicit", "ros2"] if mechanism == "h2_air_9" else ["off", "explicit"])
        nx = _side(rng, 8, 72)
        ny, nz = (max(6, int(nx * rng.uniform(0.6, 1.1))) for _ in range(2))
        cells = nx * ny * nz
        records = precision == "fp64" and chem != "ros2" and cells < 1.5e5
        return _mc("slab", nx, ny, nz, _steps(cells, 1.2e7, 100), "records" if records else "fields",
                   mechanism=mechanism, chem=chem, precision=precision)
    if flow == "inflow":
        return _mc("inflow", _side(rng, 32, 80), _side(rng, 8, 48), _side(rng, 8, 48), rng.randint(40, 100), "fields",
                   precision=rng.choice(["fp64", "fp32"]), restart=True)
    if flow == "flame":
        return _mc("flame", _side(rng, 64, 512), _side(rng, 8, 16), _side(rng, 8, 16), rng.randint(50, 150), "fields",
                   chem=rng.choice(["explicit", "ros2"]), precision="fp32", restart=True)
    if flow == "turbulence":
        n = _side(rng, 24, 64)
        return _mc("turbulence", n, n, n, rng.randint(15, 40), "fields", chem=rng.choice(["ros2", "explicit"]),
                   precision="fp32", restart=True)
    return dict(flow="surrogate", rows=_side(rng, 20000, 200000), batch=64 * rng.choice([8, 16, 33, 64]))


def _setup(case, seed):
    """The set-up records of a case and its Lattice keywords."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    seed = int(seed) + 1
    if case["flow"] == "tgv":
        cells, p = workloads.tgv_sc(nx, NY=ny, NZ=nz, Re=case["re"], seed=seed)
        return cells, None, dict(nu=p["nu"], gas_const=p["R"], gamma=p["gamma"], prtl=p["prtl"])
    if case["flow"] == "channel":
        cells, p = workloads.channel_sc(nx, ny, nz, seed=seed)
        return cells, None, dict(nu=p["nu"], gas_const=p["R"], gamma=p["gamma"], prtl=p["prtl"])
    m = _MECHS[case["mechanism"]]()
    fuel, y_fuel = _FUEL[case["mechanism"]]
    units = workloads.FLAME_UNITS
    if case["flow"] == "slab":
        hot = 1000.0 if case["chem"] == "off" else 1800.0
        mix, sp = workloads.mixing_layer_mc(m, nx, NY=ny, NZ=nz, T_hi=hot, fuel=fuel, Y_H2=y_fuel, seed=seed)
    elif case["flow"] == "inflow":
        mix, sp = workloads.inflow_layer_mc(m, nx, ny, nz, seed=seed)
    elif case["flow"] == "flame":
        mix, sp = workloads.flame_channel_mc(m, nx, ny, nz, seed=seed)
    else:
        # a quarter of the headline's velocity: the coarser lattices keep it stable over a pass
        mix, sp = workloads.turbulent_layer_mc(m, nx, u_rms=0.005, seed=seed)
        units = workloads.TURB_UNITS
    prec = lbmgpu.FP32 if case["precision"] == "fp32" else lbmgpu.FP64
    return mix, sp, dict(mech=m, dtype=workloads.MIXTURE_MC, species_dtype=workloads.SPECIES, dx_dt=units,
                         chem=_CHEM[case["chem"]], precision=prec)


def _surrogate_params(rng):
    """The network before its training: weights by fan-in, the standardisation of the inputs below."""
    parts = []
    for out, fan in ((128, 12), (128, 128), (128, 128), (10, 128)):
        parts += [rng.uniform(-1, 1, (out, fan)) * math.sqrt(6.0 / fan), rng.uniform(-0.1, 0.1, out)]
    parts += [np.zeros(12), np.ones(12), np.full(12, -1e9), np.full(12, 1e9), np.zeros(10), np.ones(10)]
    return np.concatenate([p.reshape(-1) for p in parts]).astype(np.float32)


def prepare(case, seed):
    if case["flow"] == "surrogate":
        rng = np.random.default_rng(seed)
        m = mech.h2_air_9()
        lat = lbmgpu.Lattice(10, 10, 10, mech=m, dtype=workloads.MIXTURE_MC, species_dtype=workloads.SPECIES,
                             dx_dt=workloads.FLAME_UNITS, chem=lbmgpu.CHEM_ROSENBROCK)
        x = rng.standard_normal((case["rows"], 12), dtype=np.float32)
        a = rng.standard_normal((12, 10)).astype(np.float32) / 3.0
        y = np.tanh(x @ a) + 0.05 * rng.standard_normal((case["rows"], 10), dtype=np.float32)
        lat.surrogate_params(_surrogate_params(rng))
        lat.surrogate_load_samples(x, y)
        return dict(case=case, lat=lat, x=x)
    cells, species, kw = _setup(case, seed)
    lat = lbmgpu.Lattice(*cells.shape, **kw)
    state = dict(case=case, lat=lat, cells=cells, species=species)
    if species is not None and case["out"] == "records":
        # one array for all species, so that their records come back as one output per field
        state["all"] = np.stack(species)
        state["species"] = list(state["all"])
    if case["out"] == "fields":
        planes = 10 + 2 * lat.ns if lat.ns else 9  # a single component fills 7 of them
        state["fields"] = np.zeros(planes * cells.size, np.float32)
    if not case.get("restart"):
        lat.upload(cells, state["species"])
        lat.init()
        lat.synchronize()
    return state


def run(state):
    case, lat = state["case"], state["lat"]
    if case["flow"] == "surrogate":
        loss = lat.surrogate_train(epochs=1, batch=case["batch"], lr=1e-3, seed=1)
        return {"loss": loss, "params": lat.surrogate_params(), "grads": lat.surrogate_grads(),
                "predictions": lat.surrogate_eval(state["x"])}
    if case.get("restart"):
        lat.upload(state["cells"], state["species"])
        lat.init()
    lat.step(case["steps"])
    if case["out"] == "fields":
        out = state["fields"]
        rc = lat.L.lbmgpu_vtk_fields(lat.h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                                     ctypes.c_size_t(out.size), 0)
        if rc < 0:
            raise lbmgpu.LbmGpuError(rc, "lbmgpu_vtk_fields")
        return out if lat.ns else out[: 7 * state["cells"].size]
    cells, species = state["cells"], state["species"]
    lat.download(cells, species)
    got = {name: cells[name] for name in cells.dtype.names if name != "type"}
    if species is not None:
        got["species"] = {name: state["all"][name] for name in state["all"].dtype.names}
    return got


def work(case):
    """Each population and the temperature read once and written once per time step, and the records or
    fields of the pass; operations as the model's formulas count them per cell."""
    if case["flow"] == "surrogate":
        flops = 2.0 * (12 * 128 + 2 * 128 * 128 + 128 * 10) * case["rows"]
        return {"bytes": case["rows"] * (3 * 12 + 2 * 10) * 4.0 + 5 * 36046 * 4.0, "flops": 4.0 * flops}
    cells = float(case["nx"] * case["ny"] * case["nz"])
    ghosts = float((case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2))
    if "mechanism" not in case:
        size, record, fields, per_step = 54 * 8, 1024, 7, 1200.0
    else:
        ns = 9 if case["mechanism"] == "h2_air_9" else 6
        size = 27 * (ns + 1) * (4 if case["precision"] == "fp32" else 8) + 8
        record, fields = 600 + 472 * ns, 10 + 2 * ns
        per_step = 27.0 * (ns + 1) * 25 + 60.0 * ns * ns
        per_step += {"off": 0.0, "explicit": 2500.0, "ros2": 8000.0}[case["chem"]]
    moved = 2.0 * size * cells * case["steps"]
    moved += ghosts * (record if case["out"] == "records" else 4 * fields)
    moved += ghosts * record if case.get("restart") else 0.0
    return {"bytes": moved, "flops": per_step * cells * case["steps"]}


# ---- the single-component model in 64 bits, in plain torch -------------------------------------
_C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
      (1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1),
      (0, -1, 1), (1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)]


def _psi(u, z):
    return [1 - z, (z + u) / 2, (z - u) / 2]


def _feq(rho, u, theta, corr):
    F = [_psi(u[a], theta + u[a] ** 2 + corr[a]) for a in range(3)]
    return torch.stack([rho * F[0][c[0]] * F[1][c[1]] * F[2][c[2]] for c in _C])


def _geq(rho, U, theta, u):
    P = [_psi(u[a], theta + u[a] ** 2) for a in range(3)]
    A = []
    for a in range(3):
        s, t = theta ** 2 + 2 * theta * u[a] ** 2, theta * u[a]
        A.append([-s, (t + s) / 2, (s - t) / 2])
    E = U + (u[0] ** 2 + u[1] ** 2 + u[2] ** 2) / 2
    return torch.stack([rho * (E * P[0][i] * P[1][j] * P[2][k] + A[0][i] * P[1][j] * P[2][k]
                               + P[0][i] * A[1][j] * P[2][k] + P[0][i] * P[1][j] * A[2][k]) for i, j, k in _C])


def _moments(f, g, R, cv):
    c = torch.tensor(_C, dtype=torch.float64, device=f.device)
    rho = f.sum(0)
    u = torch.einsum("lxyz,la->axyz", f, c) / rho
    P = torch.einsum("lxyz,la,lb->abxyz", f, c, c)
    rhoe = g.sum(0)
    T = (rhoe / rho - (u ** 2).sum(0) / 2) / cv
    return dict(rho=rho, u=u, P=P, rhoe=rhoe, T=T, p=rho * R * T, q=torch.einsum("lxyz,la->axyz", g, c))


def exact(case, seed):
    """The periodic single-component box; the other flows' boundary closures, gas properties (rounded to
    single precision at every change of units) and adaptive chemistry have no short restatement."""
    if case["flow"] != "tgv" or case["nx"] * case["ny"] * case["nz"] * case["steps"] > 4.5e8:
        return None
    cells, _, kw = _setup(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    R, gamma = kw["gas_const"], kw["gamma"]
    cv = R / (gamma - 1)
    cp = cv + R
    inner = (slice(1, -1),) * 3
    get = lambda name: torch.tensor(np.ascontiguousarray(cells[name][inner]), device=dev)  # noqa: E731
    T, p, u = get("temp"), get("p"), torch.stack([get("u"), get("v"), get("w")])
    rho = p / (R * T)
    theta, zero = R * T, torch.zeros_like(u)
    # the start: populations at rest, the energy set from its moments
    f = _feq(rho, zero, theta, zero)
    rhoe, H = rho * cv * T, cp * T
    q, r = H * rho * u, H * p
    g = []
    for c in _C:
        val = rhoe + sum(q[a] * c[a] for a in range(3)) / theta
        val = val + sum((r - rhoe * theta) * (c[a] * c[a] - theta) for a in range(3)) / (2 * theta ** 2)
        for a in range(3):
            val = val * (theta / 2 if c[a] else 1 - theta)
        c2 = c[0] ** 2 + c[1] ** 2 + c[2] ** 2
        b = 3.0 if c2 == 0 else (-0.5 if c2 == 1 else 0.0)
        g.append(val + b * ((1 - 3 * theta) / (2 * theta) * (r - theta * rhoe)))
    g = torch.stack(g)
    eye = torch.eye(3, dtype=torch.float64, device=dev)[:, :, None, None, None]
    m = dict(rho=rho, u=u, P=p * eye, rhoe=rhoe, T=T, p=p)
    fpc = gpc = None
    for _ in range(case["steps"]):
        rho, u, T, p = m["rho"], m["u"], m["T"], m["p"]
        theta, mu = R * T, kw["nu"] * rho
        kappa = mu * cp / kw["prtl"]
        om1, om = 2 * p * cp / (p * cp + 2 * kappa), 2 * p / (p + 2 * mu)
        # face differences; next to a periodic ghost plane they are one-sided where the far side is
        # fluid, as the reference's stencil takes them
        Q = rho * u * (1 - 3 * R * T) - rho * u ** 3
        dQ = torch.empty_like(Q)
        for a in range(3):
            x = Q[a].movedim(a, 0)
            d = torch.empty_like(x)
            d[1:-1] = (x[2:] - x[:-2]) / 2
            d[0], d[-1] = x[1] - x[0], x[-1] - x[-2]
            dQ[a] = d.movedim(0, a)
        Peq = p * eye + rho * u[:, None] * u[None]
        dq = torch.einsum("axyz,abxyz->bxyz", u, m["P"] - Peq) + u * dQ / 2
        fpc = f + om * (_feq(rho, u, theta, (2 - om) / (2 * rho * om) * dQ) - f)
        geq = _geq(rho, m["rhoe"] / rho - (u ** 2).sum(0) / 2, theta, u)
        gpc = g + om1 * (geq - g)
        for i, c in enumerate(_C):
            if c[0] ** 2 + c[1] ** 2 + c[2] ** 2 == 1:
                gpc[i] -= (om - om1) * sum(c[a] * dq[a] for a in range(3)) / 2
        f = torch.stack([torch.roll(fpc[i], c, (0, 1, 2)) for i, c in enumerate(_C)])
        g = torch.stack([torch.roll(gpc[i], c, (0, 1, 2)) for i, c in enumerate(_C)])
        m = _moments(f, g, R, cv)
    h = lambda t: t.cpu().numpy()  # noqa: E731
    fields = dict(rho=h(m["rho"]), temp=h(m["T"]), p=h(m["p"]), u=h(m["u"][0]), v=h(m["u"][1]), w=h(m["u"][2]))
    for name, value in fields.items():
        cells[name][inner] = value
    if case["out"] == "fields":
        flat = lambda a: np.asarray(a, np.float64).transpose(2, 1, 0).reshape(-1)  # noqa: E731
        vel = np.stack([flat(cells[k]) for k in "uvw"], -1).reshape(-1)
        return np.concatenate([flat(cells["rho"]), vel, flat(cells["type"]), flat(cells["temp"]), flat(cells["p"])])
    for name, value in dict(f=f, g=g, fpc=fpc, gpc=gpc, energy_flux=m["q"]).items():
        cells[name][inner] = h(value).transpose(1, 2, 3, 0)
    cells["p_tensor"][inner] = h(m["P"]).transpose(2, 3, 4, 0, 1)
    cells["rhoe"][inner] = h(m["rhoe"])
    return {name: cells[name].astype(np.float64) for name in cells.dtype.names if name != "type"}
