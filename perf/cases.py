"""Performance cases of the marker-in-cell framework: the calls its programs make, over the sizes
they make them at.

Boxes, grids and marker counts are those of `fvmic2d_gb300.workloads`, the tests and `bench.py`
(64 x 64 convection, 1024 x 256 visco-elasto-plastic, 1024 x 1024 ice, 128 x 32 and 512 x 128
subduction), with odd and ragged sizes between them.  The kinds of case:

  cycle       the marker work between one host solve and the next (stress and strain update,
              sub-grid diffusion, advection, binning, yielding, projection); returns the nodal
              fields the next solve reads, which every marker column of the cycle enters
  ensemble    one captured step of independent members side by side
  handover    a host program's step: markers and solver fields up, one step, everything down
  solve       the direct solve of an assembled Stokes or thermal system
  timestep    one whole time step of the subduction program, solves included
  train       training of the learned creep closure (forward and backward passes)

The flows are closed cells (no marker leaves through a wall), so that a box can be stepped for as
long as a program steps it.
"""
import ctypes
import math

import numpy as np
import torch

from fvmic2d_gb300 import gpu
from fvmic2d_gb300 import workloads as W
from fvmic2d_gb300.mic_types import MARKER_DTYPE

# nodal fields a cycle or a step leaves for the solves (projections, residual, stress changes)
NODAL_OUT = ["rho", "etaN", "etaS", "kThermal", "Cp", "lastT", "soxx", "soyy", "soxy", "dsxx", "dsyy", "dsxy", "srr"]
# nodal fields a host Stokes and thermal solve hands over each step
SOLVER_FIELDS = ["vx", "vy", "p", "edotxx", "edotyy", "edotxy", "wxy", "dsxx", "dsyy", "dsxy", "thisT"]
MARKER_OUT = ["X", "Y", "VX", "VY", "T", "Tdot", "sxx", "syy", "sxy", "eta", "mu", "rho", "p", "exx", "eyy", "exy",
              "Eii", "wxy", "srr", "Mat", "cellX", "cellY"]
# algorithmic bytes of one step: 436 per marker, 352 per node; about 520 double-precision
# operations per marker (the law-7 solve adds about 180)
STEP_MARKER_BYTES, STEP_NODE_BYTES, STEP_MARKER_FLOPS, LAW7_FLOPS = 436, 352, 520, 180


def listed():
    return [
        # the smallest box a program steps: launches and latency count
        {"name": "convection_64", "kind": "cycle", "box": "convection", "nx": 64, "ny": 64, "nm": 4},
        # two-material visco-elasto-plastic production box
        {"name": "vep_1024x256", "kind": "cycle", "box": "vep", "nx": 1024, "ny": 256, "nm": 4},
        # the largest box, composite creep through the learned closure on the tensor cores
        {"name": "ice_surrogate_1024", "kind": "cycle", "box": "ice", "mode": 2, "plastic": False,
         "nx": 1024, "ny": 1024, "nm": 4},
        # a ragged ice box that yields, with the exact creep solve, 9 markers a cell
        {"name": "ice_exact_333x517", "kind": "cycle", "box": "ice", "mode": 0, "plastic": True, "nx": 333,
         "ny": 517, "nm": 3},
        # a box periodic in x, odd sizes, 25 markers a cell
        {"name": "periodic_509x127", "kind": "cycle", "box": "periodic", "nx": 509, "ny": 127, "nm": 5},
        # a parameter study: independent convection runs stepped as one captured graph
        {"name": "ensemble_12", "kind": "ensemble", "members": 12},
        # a host program that keeps the markers: everything crosses the bus each step
        {"name": "handover_256x64", "kind": "handover", "nx": 256, "ny": 64, "nm": 4},
        # the direct solves of the subduction program, at its two sizes
        {"name": "stokes_128x32", "kind": "solve", "system": "stokes", "nx": 128, "ny": 32},
        {"name": "stokes_512x128", "kind": "solve", "system": "stokes", "nx": 512, "ny": 128},
        {"name": "thermal_512x128", "kind": "solve", "system": "thermal", "nx": 512, "ny": 128},
        # the subduction program's time step: plasticity iterations around the solves
        {"name": "subduction_128x32", "kind": "timestep", "nx": 128, "ny": 32, "nm": 4},
        # training of the creep closure from scratch
        {"name": "train_4096", "kind": "train", "samples": 262144, "batch": 4096, "steps": 200},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _subduction_grid(rng, most):
    """four cells along x for one along y, a few more or less, on grids where no pressure cell is
    cut off between slab and plate (there the Stokes matrix is singular)"""
    ny = 4 * _log_int(rng, 6, most)
    return 4 * ny + rng.choice([-3, 0, 1]), ny


def draw(rng):
    kind = rng.choice(["cycle", "cycle", "cycle", "cycle", "ensemble", "handover", "solve", "solve", "timestep",
                       "train"])
    if kind == "cycle":
        box = rng.choice(["convection", "vep", "ice", "ice", "periodic"])
        lo, hi = {"convection": (40, 400), "vep": (64, 640), "ice": (64, 640), "periodic": (64, 512)}[box]
        nx = _log_int(rng, lo, hi)
        ny = _log_int(rng, 32, 256) if box != "periodic" else _log_int(rng, 24, 128)
        c = {"kind": kind, "box": box, "nx": nx, "ny": ny, "nm": rng.choice([3, 4, 5])}
        if box == "ice":
            c["mode"], c["plastic"] = rng.choice([0, 2, 2]), rng.random() < 0.5
        return c
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 12)}
    if kind == "handover":
        return {"kind": kind, "nx": _log_int(rng, 64, 384), "ny": _log_int(rng, 24, 96), "nm": rng.choice([3, 4])}
    if kind == "solve":
        system = rng.choice(["stokes", "thermal"])
        if system == "thermal":
            return {"kind": kind, "system": system, "nx": _log_int(rng, 64, 512), "ny": _log_int(rng, 24, 128)}
        nx, ny = _subduction_grid(rng, 28)
        return {"kind": kind, "system": system, "nx": nx, "ny": ny}
    if kind == "timestep":
        nx, ny = _subduction_grid(rng, 11)
        return {"kind": kind, "nx": nx, "ny": ny, "nm": rng.choice([3, 4])}
    return {"kind": kind, "samples": rng.choice([65536, 131072, 262144]), "batch": 128 * _log_int(rng, 8, 64),
            "steps": rng.randint(60, 240)}


# ---- preparation -----------------------------------------------------------------------


class _Device:
    """A library-owned device array as torch sees it (no copy); keeps its context alive."""

    def __init__(self, P, ptr, shape):
        self.context = P
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _view(P, name):
    p = ctypes.POINTER(ctypes.c_double)()
    P._check(P.L.mic_nodal_device_ptr(P.h, gpu.NF[name], ctypes.byref(p)), "mic_nodal_device_ptr")
    return torch.as_tensor(_Device(P, ctypes.cast(p, ctypes.c_void_p).value, (P.NY, P.NX)), device="cuda")


def _closed_flow(wl, speed):
    """one closed convection cell on the workload's grid, with its strain rates and vorticity"""
    g = wl.grid
    pi, LX, LY, a = math.pi, g.LX, g.LY, speed
    b = a * LY / LX
    sx, cx, sy, cy = (lambda v, L, f=f: f(pi * v / L) for f in (np.sin, np.cos, np.sin, np.cos))
    X, YC = np.meshgrid(g.x, g.yc[1:])
    XC, Y = np.meshgrid(g.xc[1:], g.y)
    Xc, Yc = np.meshgrid(g.xc[: g.NX], g.yc[: g.NY])
    Xb, Yb = np.meshgrid(g.x, g.y)
    exx = a * pi / LX * cx(Xc, LX) * cy(Yc, LY)
    dvxdy = -a * pi / LY * sx(Xb, LX) * sy(Yb, LY)
    dvydx = b * pi / LX * sx(Xb, LX) * sy(Yb, LY)
    f = {"vx": a * sx(X, LX) * cy(YC, LY), "vy": -b * cx(XC, LX) * sy(Y, LY), "edotxx": exx, "edotyy": -exx,
         "edotxy": 0.5 * (dvxdy + dvydx), "wxy": 0.5 * (dvxdy - dvydx)}
    wl.nodal.update(f)
    dt = 0.5 * min(float(np.min(np.diff(g.x))), float(np.min(np.diff(g.y)))) / (a + b)
    wl.dt = wl.dt_thermal = dt


def _stresses(wl, eta):
    n = wl.nodal
    for s, e in (("xx", "edotxx"), ("yy", "edotyy"), ("xy", "edotxy")):
        n["so" + s] = 2.0 * eta * n[e]
        n["ds" + s] = 0.05 * n["so" + s]


_NETS = {}


def _network(P):
    """the trained closure a program keeps: one network, trained once"""
    if not _NETS:
        P.creep_train(nsamples=1 << 19, batch=4096, steps=4000, seed=1)
        _NETS["params"] = P.creep_params()
    P.creep_set_params(_NETS["params"])


def _box(case, seed):
    """a box with its markers on the device, and its grain sizes (ice) -- before the first cycle"""
    box, nx, ny, nm = case.get("box", "vep"), case["nx"], case["ny"], case["nm"]
    rng = np.random.default_rng(seed)
    if box == "vep":  # markers as the set-up of a host program leaves them
        wl = W.vep_slab_box(nx, ny, nm, seed % 100003)
        _closed_flow(wl, 1e-9 * rng.uniform(0.5, 2.0))
        _stresses(wl, 1e21)
        P = gpu.MicProblem(wl)
        return wl, P, None
    if box == "periodic":
        wl = W.periodic_box(nx, ny, nm, seed % 100003)
        return wl, gpu.MicProblem(wl), None
    if box == "convection":
        wl = W.convection_member(nx, ny, nm, nm, 10 ** rng.uniform(4, 6), 10 ** rng.uniform(1, 4), seed % 100003)
    else:
        wl = W.ice_member(nx, ny, seed % 100003, nm)
        wl.materials.hasPlasticity[0] = int(case["plastic"])
        shape = (ny + 1, nx + 1)
        wl.nodal["lastT"] = 100.0 + 153.0 * wl.grid.y[:, None] / wl.grid.LY + 20.0 * rng.random(shape)
        wl.nodal["thisT"] = wl.nodal["lastT"] + 0.5 * rng.random(shape)
        wl.nodal["p"] = 1e8 * rng.random(shape)
        for c in ("xx", "yy", "xy"):  # stresses of an ice shell, 100 Pa to 100 kPa, and their changes
            wl.nodal["so" + c] = rng.choice([-1.0, 1.0], shape) * 10.0 ** rng.uniform(2, 5, shape)
            wl.nodal["ds" + c] = 0.01 * wl.nodal["so" + c]
    P = gpu.MicProblem(wl, capacity=wl.capacity)
    gpu.initialize_markers(P, nm, nm, seed=seed % 100003)
    grain = None
    if box == "ice":
        grain = 10.0 ** (-4.0 + 3.0 * rng.random(P.n))
        P.set_grain_size(grain)
        P.projectNodalFieldToMarkersS("p", "p")
        for c in ("xx", "yy", "xy"):
            P.projectNodalFieldToMarkersS("so" + c, "s" + c)
        for f in ("exx", "exy"):  # strain rates over eight decades, by the node
            P.set_nodal("heating", 10.0 ** rng.uniform(-18, -10, (ny + 1, nx + 1)))
            P.projectNodalFieldToMarkersS("heating", f)
        if case["mode"]:
            _network(P)
        P.creep_configure(mode=case["mode"], tol=2e-14, maxit=60, polish_iters=3, polish_tol=1e-7)
    return wl, P, grain


def _pre(P, dt):
    y, t = ctypes.c_int(0), ctypes.c_double(0.0)
    P._check(P.L.mic_step_pre_stokes(P.h, dt, ctypes.byref(y), ctypes.byref(t)), "mic_step_pre_stokes")
    return y.value, t.value


def _members(case, seed):
    """grids and resolutions as the convection ensemble mixes them"""
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["members"])  # the work depends on the case alone
    wls = []
    for k in range(case["members"]):
        n, nm = int(sizes.choice([64, 64, 96, 128])), int(sizes.integers(3, 6))
        wls.append(W.convection_member(n, n, nm, nm, 10 ** rng.uniform(4, 6), 10 ** rng.uniform(1, 4),
                                       (seed * 31 + k) % 100003))
    return wls


def _assembled(case, seed):
    """the subduction box with its systems' inputs projected and the system assembled"""
    wl, topt = W.subduction_box(nx_cells=case["nx"], ny_cells=case["ny"], nm=2, seed=seed % 100003)
    P = gpu.MicProblem(wl)
    P.findMarkerCells()
    P.updateMarkerRho()
    P.projectMarkersNodesAll2()
    if case["system"] == "stokes":
        P.formVEPSystem(topt.sub, topt.dtMax)
    else:
        P.enforceThermalBCs1(topt.sub)
        P.formThermalSystem(topt.sub, topt.dtMax)
    return P


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cycle":
        wl, P, _ = _box(case, seed)
        _pre(P, wl.dt)
        return {"kind": kind, "P": P, "dt": wl.dt, "views": {f: _view(P, f) for f in NODAL_OUT}}
    if kind == "ensemble":
        wls = _members(case, seed)
        ps = []
        for wl in wls:
            P = gpu.MicProblem(wl, capacity=wl.capacity)
            gpu.initialize_markers(P, *wl.nm, seed=wl.seed)
            ps.append(P)
        dts = np.array([wl.dt for wl in wls])
        return {"kind": kind, "E": gpu.MicEnsemble(ps), "dts": dts,
                "views": [{f: _view(P, f) for f in ("lastT", "etaN", "soxx", "soyy", "soxy")} for P in ps]}
    if kind == "handover":
        wl, P, _ = _box(case, seed)
        return {"kind": kind, "P": P, "dt": wl.dt, "markers": P.markers,
                "solver": {f: np.ascontiguousarray(wl.nodal[f]) for f in SOLVER_FIELDS}}
    if kind == "solve":
        P = _assembled(case, seed)
        return {"kind": kind, "P": P, "which": P.STOKES if case["system"] == "stokes" else P.THERMAL}
    if kind == "timestep":
        wl, topt = W.subduction_box(nx_cells=case["nx"], ny_cells=case["ny"], nm=case["nm"], seed=seed % 100003)
        topt.densityControl = 1  # as the program runs; firstStep is 1 in its first step alone
        topt.density.NMX = topt.density.NMY = case["nm"]
        for f in ("slabAngle", "slabAge", "overridingPlateThickness", "rootThickness", "rootCenter", "rootWidth"):
            setattr(topt.density, f, getattr(topt.sub, f))
        topt.firstStep = 0
        topt.maxNumPlasticity = 2  # every pass the same work: two plasticity iterations
        P = gpu.MicProblem(wl, capacity=2 * len(wl.markers))
        return {"kind": kind, "P": P, "topt": topt, "t": 0.0,
                "views": {f: _view(P, f) for f in ("vx", "vy", "p", "thisT", "rho", "etaS", "soxx", "soxy")}}
    wl = W.convection_member(4, 4, 2, 2, 1e4, 10.0, 1)  # training needs a context, no markers
    return {"kind": kind, "P": gpu.MicProblem(wl, capacity=64), "seed": seed % 100003 + 1,
            "args": {k: case[k] for k in ("samples", "batch", "steps")}}


# ---- one pass --------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "cycle":
        P, dt = state["P"], state["dt"]
        res, smax = ctypes.c_double(0.0), ctypes.c_double(0.0)
        P._check(P.L.mic_step_post_stokes(P.h, dt, 1, ctypes.byref(res)), "mic_step_post_stokes")
        P._check(P.L.mic_step_post_thermal(P.h, dt, ctypes.byref(smax)), "mic_step_post_thermal")
        yielding, tmax = _pre(P, dt)
        return {"nodal": state["views"], "residual": res.value, "max_abs_sxx": smax.value, "max_T": tmax,
                "yielding": yielding}
    if kind == "ensemble":
        E = state["E"]
        E.step(state["dts"], state["dts"], 1, graph=True)
        E.synchronize()
        return {"nodal": state["views"]}
    if kind == "handover":
        P = state["P"]
        P.upload_markers(state["markers"])
        for f, v in state["solver"].items():
            P.set_nodal(f, v)
        _, res = P.step(state["dt"], state["dt"], True)
        m = P.markers
        return {"markers": {f: m[f] for f in MARKER_OUT}, "nodal": {f: P.get_nodal(f) for f in NODAL_OUT},
                "residual": res}
    if kind == "solve":
        P = state["P"]
        P.linear_solve(state["which"])
        return P.solution(state["which"])
    if kind == "timestep":
        rep = state["P"].subductionTimestep(state["topt"], state["t"])
        state["t"] += rep["dt"]
        return {"nodal": state["views"], "report": rep}
    a = state["args"]
    loss = state["P"].creep_train(nsamples=a["samples"], batch=a["batch"], steps=a["steps"], seed=state["seed"])
    return {"loss": loss, "params": state["P"].creep_params()}


# ---- work ------------------------------------------------------------------------------


def _step_work(n, nodes, law7):
    return {"bytes": n * STEP_MARKER_BYTES + nodes * STEP_NODE_BYTES,
            "flops": n * (STEP_MARKER_FLOPS + (LAW7_FLOPS if law7 else 0))}


def _lu_work(nx, ny, system):
    """banded elimination at its least: n kl (kl + ku) multiply-adds without pivoting's fill;
    the band read and written once"""
    dof = 3 if system == "stokes" else 1
    n = dof * (nx + 1) * (ny + 1)
    kl = dof * (min(nx, ny) + 2) + (2 if dof == 3 else -1)
    return {"bytes": 16.0 * n * (2 * kl + 1), "flops": 2.0 * n * kl * kl}


def work(case):
    kind = case["kind"]
    if kind in ("cycle", "handover"):
        n = case["nx"] * case["ny"] * case["nm"] ** 2
        nodes = (case["nx"] + 1) * (case["ny"] + 1)
        w = _step_work(n, nodes, case.get("box") == "ice")
        if kind == "handover":  # the records up and down once
            w["bytes"] += 2 * n * MARKER_DTYPE.itemsize
        return w
    if kind == "ensemble":
        ws = [_step_work(wl.capacity, wl.grid.NX * wl.grid.NY, False) for wl in _members(case, 0)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if kind == "solve":
        return _lu_work(case["nx"], case["ny"], case["system"])
    if kind == "timestep":
        n = case["nx"] * case["ny"] * case["nm"] ** 2
        s = _step_work(n, (case["nx"] + 1) * (case["ny"] + 1), False)
        a, b = (_lu_work(case["nx"], case["ny"], k) for k in ("stokes", "thermal"))
        return {k: s[k] + 2 * a[k] + b[k] for k in ("bytes", "flops")}
    macs = 4 * 64 + 64 * 64 + 64  # forward; the backward pass is twice that
    return {"bytes": 20.0 * case["samples"] + 24.0 * case["batch"] * case["steps"],
            "flops": 6.0 * macs * case["batch"] * case["steps"] + 2000.0 * case["samples"]}


# ---- the same in plain torch, 64 bits ----------------------------------------------------


class _Plain:
    """One box stepped with plain torch operations in 64 bits (free-slip walls, material laws 0, 1,
    5 and 7, Mohr-Coulomb yielding)."""

    def __init__(self, wl, markers, grain=None):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda")
        g = wl.grid
        self.wl, self.NX, self.NY = wl, g.NX, g.NY
        self.x, self.y, self.xc, self.yc = t(g.x), t(g.y), t(g.xc), t(g.yc)
        self.f = {k: t(v).reshape(-1) for k, v in wl.nodal.items()}
        for k in NODAL_OUT + SOLVER_FIELDS:
            self.f.setdefault(k, torch.zeros(g.NX * g.NY, dtype=torch.float64, device="cuda"))
        self.m = {k: t(markers[k]) for k in MARKER_OUT}
        self.grain = None if grain is None else t(grain)

    def locate(self):
        m = self.m
        self.inside = (m["X"] >= 0) & (m["Y"] >= 0) & (m["X"] <= self.wl.grid.LX) & (m["Y"] <= self.wl.grid.LY)
        cell = lambda g, v: (torch.searchsorted(g, v, right=True) - 1).clamp(0, len(g) - 2)
        self.i, self.j = cell(self.x, m["X"]), cell(self.y, m["Y"])
        m["cellX"], m["cellY"] = (torch.where(self.inside, c, -1).double() for c in (self.i, self.j))
        self.fx, self.fy = self.frac(self.x, m["X"], self.i), self.frac(self.y, m["Y"], self.j)

    @staticmethod
    def frac(g, v, i):
        return (v - g[i]) / (g[i + 1] - g[i])

    def put(self, key, v):
        self.m[key] = torch.where(self.inside, v, self.m[key])

    def centre(self, clamp):
        X, Y = self.m["X"], self.m["Y"]
        i = self.i + (X >= self.xc[self.i + 1]).long()
        j = self.j + (Y >= self.yc[self.j + 1]).long()
        if clamp:
            i, j = i.clamp(1, self.NX - 2), j.clamp(1, self.NY - 2)
        return i, j, self.frac(self.xc, X, i), self.frac(self.yc, Y, j)

    def interp(self, f, at):
        i, j, a, b = at
        k = j * self.NX + i
        return ((1 - a) * (1 - b) * f[k] + a * (1 - b) * f[k + 1] + (1 - a) * b * f[k + self.NX]
                + a * b * f[k + self.NX + 1])

    def sums(self, i, j, w, vs):
        ok = self.inside & (i < self.NX) & (j < self.NY)
        k, w = (j * self.NX + i)[ok], w[ok]
        out = [torch.zeros(self.NX * self.NY, dtype=torch.float64, device="cuda").index_add_(0, k, w * v[ok]) for v in vs]
        return out + [torch.zeros_like(out[0]).index_add_(0, k, w)]

    def project(self, vs, at, local=False):
        i, j, a, b = at
        if local:
            ox, oy = a >= 0.5, b >= 0.5
            s = self.sums(i + ox.long(), j + oy.long(), torch.where(ox, a, 1 - a) * torch.where(oy, b, 1 - b), vs)
        else:
            s = None
            for ox in (0, 1):
                for oy in (0, 1):
                    r = self.sums(i + ox, j + oy, (a if ox else 1 - a) * (b if oy else 1 - b), vs)
                    s = r if s is None else [p + q for p, q in zip(s, r)]
        return [torch.where(s[-1] != 0, v / s[-1], torch.zeros_like(v)) for v in s[:-1]]

    def basic(self):
        return self.i, self.j, self.fx, self.fy

    def creep(self, edot):
        """stress at which the composite law gives the strain rate, by bisection of ln s"""
        m, R = self.m, 8.3144621
        T, d, P = m["T"], self.grain, m["p"].clamp(min=1.0)
        Vm, b = 1.97e-5, 4.52e-10
        lin = 42.0 * Vm / (R * T * d * d) * (9.10e-4 * torch.exp(-59.4e3 / (R * T))
                                             + math.pi * 2.0 * b / d * 5.8e-4 * torch.exp(-49e3 / (R * T)))
        arr = lambda Q: torch.exp((-Q - 13e-6 * P) / (R * T))
        gbs = torch.where(T < 255, 3.9e-3 * arr(49e3), 3.0e26 * arr(192e3)) / d ** 1.4
        dis = torch.where(T < 258, 4.0e5 * arr(60e3), 6.0e28 * arr(180e3))
        bas = 5.5e7 * arr(60e3)

        def rate(s):
            x = s / 1e6
            return lin * s + 1.0 / (1.0 / (bas * x ** 2.4) + 1.0 / (gbs * x ** 1.8)) + dis * x ** 4.0

        top = edot / lin
        lo, hi = torch.zeros_like(top), torch.log(top.clamp(min=1.0))
        for _ in range(64):
            mid = 0.5 * (lo + hi)
            over = rate(torch.exp(mid)) > edot
            lo, hi = torch.where(over, lo, mid), torch.where(over, mid, hi)
        s = torch.exp(0.5 * (lo + hi))
        s = torch.where(rate(torch.ones_like(s)) >= edot, torch.ones_like(s), s)
        s = torch.where(top < 1.0, top, s)
        return torch.where(edot > 0, s / (2.0 * edot), 0.5 / lin)

    def rheology(self, dt):
        m, M, O = self.m, self.wl.materials, self.wl.options
        eii = torch.sqrt(0.5 * (m["exx"] ** 2 + m["eyy"] ** 2) + m["exy"] ** 2)
        X = m["eta"] / (m["mu"] * dt + m["eta"])
        sv = [m["s" + c] * X + 2 * m["eta"] * m["e" + c] * (1 - X) for c in ("xx", "yy", "xy")]
        sii = torch.sqrt(0.5 * (sv[0] ** 2 + sv[1] ** 2) + sv[2] ** 2)
        old, new, mu = m["eta"], m["eta"].clone(), m["mu"].clone()
        for k in range(M.nMaterials):
            of = m["Mat"] == k
            law, e0, Q = M.hasEtaT[k], M.materialEta[k], M.QonR[k]
            eta = {0: lambda: torch.full_like(old, e0), 1: lambda: e0 * torch.exp(Q * (1 / m["T"] - 1 / M.Tref[k])),
                   5: lambda: e0 * torch.exp(-Q * m["T"]), 7: lambda: self.creep(eii)}[law]()
            mu = torch.where(of, torch.full_like(mu, M.materialMu[k]), mu)
            if M.hasPlasticity[k] == 1:
                sy = (M.materialCohesion[k] + M.materialFriction[k] * m["p"]).clamp(min=0.0)
                y = of & self.inside & (sii > sy)
                ey = torch.maximum(sy / 2 / eii, O.fractionalEtamin * eta).clamp(O.etamin, O.etamax)
                sio = torch.sqrt(0.5 * (m["sxx"] ** 2 + m["syy"] ** 2) + m["sxy"] ** 2)
                scale = torch.where(y & (sio != 0), sy / sio, torch.ones_like(sy))
                for c in ("sxx", "syy", "sxy"):
                    m[c] = m[c] * scale
                self.yielding = self.yielding or bool(y.any())
                eta = torch.where(y, ey, old)
            new = torch.where(of, eta, new)
        self.put("eta", new)
        self.put("mu", mu)
        m["eta"] = m["eta"].clamp(O.etamin, O.etamax)

    def pre(self, dt):
        m, M = self.m, self.wl.materials
        self.locate()
        prop = lambda a: torch.as_tensor(np.array(a[:]), device="cuda")[m["Mat"].long().clamp(min=0)]
        self.put("rho", -prop(M.materialRho) * (prop(M.materialAlpha) * m["T"]))
        self.max_T = float(m["T"][self.inside].max())
        self.yielding = False
        self.rheology(dt)
        f = self.f
        at, ct = self.basic(), self.centre(False)
        f["rho"], f["etaS"], f["kThermal"], f["lastT"], f["Cp"] = self.project(
            [m["rho"], m["eta"], prop(M.materialkThermal), m["T"], prop(M.materialCp)], at)
        f["etaN"], = self.project([m["eta"]], ct)
        f["soxx"], f["soyy"] = self.project([m["sxx"], m["syy"]], ct, local=True)
        f["soxy"], = self.project([m["sxy"]], at, local=True)

    def post(self, dt):
        m, f, D = self.m, self.f, self.wl.options.subgridStressDiffusivity
        at, ct = self.basic(), self.centre(True)
        gc, gb = (lambda k: self.interp(f[k], ct)), (lambda k: self.interp(f[k], at))
        self.put("p", gc("p"))
        self.put("wxy", gb("wxy"))
        for e, so, ds, g in (("exx", "soxx", "dsxx", gc), ("eyy", "soyy", "dsyy", gc), ("exy", "soxy", "dsxy", gb)):
            self.put(e, g(so) / 2 / m["eta"] + g(ds) / 2 / dt / m["mu"])
        self.put("srr", torch.sqrt((m["exx"] - gc("edotxx")) ** 2 + (m["exy"] - gb("edotxy")) ** 2))
        srr, = self.project([m["srr"]], self.centre(False))
        area = torch.zeros(self.NY, self.NX, dtype=torch.float64, device="cuda")
        area[1:, 1:] = torch.diff(self.y)[:, None] * torch.diff(self.x)[None, :]
        f["srr"] = srr * area.reshape(-1)
        self.residual = float(f["srr"].sum()) / (self.wl.grid.LX * self.wl.grid.LY)
        if D > 0:
            q = 1 - torch.exp((-D * dt * m["mu"] / m["eta"]).clamp(min=-30.0))
            d = {"sxy": (gb("soxy") - m["sxy"]) * q, "sxx": (gc("soxx") - m["sxx"]) * q,
                 "syy": (gc("soyy") - m["syy"]) * q}
            for k, v in d.items():
                self.put(k, m[k] + v)
            f["dsxy"] = f["dsxy"] - self.project([d["sxy"]], at, local=True)[0]
            s = self.sums(self.i + 1, self.j + 1, (1 - (0.5 - self.fx).abs()) * (1 - (0.5 - self.fy).abs()),
                          [d["sxx"], d["syy"]])
            for k, v in (("dsxx", s[0]), ("dsyy", s[1])):
                f[k] = f[k] - torch.where(s[2] != 0, v / s[2], torch.zeros_like(v))
        for k, ds, g in (("sxx", "dsxx", gc), ("syy", "dsyy", gc), ("sxy", "dsxy", gb)):
            self.put(k, m[k] + g(ds))

    def thermal(self, dt):
        m, f = self.m, self.f
        at = self.basic()
        gb = lambda k: self.interp(f[k], at)
        dx, dy = self.x[self.i + 1] - self.x[self.i], self.y[self.j + 1] - self.y[self.j]
        diff = gb("Cp") * (self.wl.materials.materialRho[0] + gb("rho")) / gb("kThermal") / (2 / dx ** 2 + 2 / dy ** 2)
        d = (gb("lastT") - m["T"]) * (1 - torch.exp(-self.wl.options.subgridTemperatureDiffusivity * dt / diff))
        left = f["thisT"] - f["lastT"] - self.project([d], at)[0]
        d = self.interp(left, at) + d
        self.put("T", m["T"] + d)
        self.put("Tdot", d / dt)
        self.advect(dt)
        self.max_abs_sxx = float(m["sxx"][self.inside].abs().max())

    def advect(self, dt):
        m, NX, NY = self.m, self.NX, self.NY
        vx, vy, wz = self.f["vx"], self.f["vy"], self.f["wxy"]
        x, y, V = m["X"], m["Y"], []

        def sample(f, i, j, a, b):  # ghost row or column -1: free slip, the value inside
            i0, j0 = i.clamp(min=0), j.clamp(min=0)
            return ((1 - a) * (1 - b) * f[j0 * NX + i0] + a * (1 - b) * f[j0 * NX + i + 1]
                    + (1 - a) * b * f[(j + 1) * NX + i0] + a * b * f[(j + 1) * NX + i + 1])

        for s in range(4):
            i = (torch.searchsorted(self.x, x) - 1).clamp(0, NX - 2)
            j = (torch.searchsorted(self.y, y) - 1).clamp(0, NY - 2)
            jv = j - (y < self.yc[j + 1]).long()
            iv = i - (x < self.xc[i + 1]).long()
            jv, iv = jv.clamp(max=NY - 2), iv.clamp(max=NX - 2)
            fx, fy = self.frac(self.x, x, i), self.frac(self.y, y, j)
            V.append((sample(vx, i, jv, fx, self.frac(self.yc, y, jv + 1)),
                      sample(vy, iv, j, self.frac(self.xc, x, iv + 1), fy), sample(wz, i, j, fx, fy)))
            h = dt / 2 if s < 2 else dt
            x, y = m["X"] + h * V[s][0], m["Y"] + h * V[s][1]
        mean = [(a + 2 * b + 2 * c + d) / 6 for a, b, c, d in zip(*V)]
        for k, v in zip(("VX", "VY", "wxy"), mean):
            self.put(k, v)
        self.put("X", m["X"] + dt * mean[0])
        self.put("Y", m["Y"] + dt * mean[1])
        th = -mean[2] * dt
        c, s, s2, c2 = torch.cos(th), torch.sin(th), torch.sin(2 * th), torch.cos(2 * th)
        a, b, q = m["sxx"], m["syy"], m["sxy"]
        self.put("sxx", a * c * c + b * s * s - q * s2)
        self.put("syy", a * s * s + b * c * c + q * s2)
        self.put("sxy", 0.5 * (a - b) * s2 + q * c2)
        self.put("Eii", m["Eii"] + dt * torch.sqrt(0.5 * (m["exx"] ** 2 + m["eyy"] ** 2) + m["exy"] ** 2))

    def nodal(self, names):
        return {k: self.f[k].reshape(self.NY, self.NX) for k in names}


def _plain_solve(case, seed):
    P = _assembled(case, seed)
    which = P.STOKES if case["system"] == "stokes" else P.THERMAL
    rp, c, v, b = P.system(which)
    n = len(b)
    rows = torch.as_tensor(np.repeat(np.arange(n), np.diff(rp)), device="cuda")
    cols = torch.as_tensor(c.astype(np.int64), device="cuda")
    vals, rhs = torch.as_tensor(v, device="cuda"), torch.as_tensor(b, device="cuda")
    if n <= 16000:
        A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        A[rows, cols] = vals
        s = 1.0 / A.abs().amax(1)  # rows to one scale, then one step of refinement
        A, r = A * s[:, None], rhs * s
        lu, piv = torch.linalg.lu_factor(A)
        u = torch.linalg.lu_solve(lu, piv, r[:, None])
        return (u + torch.linalg.lu_solve(lu, piv, r[:, None] - A @ u))[:, 0].cpu().numpy()
    if case["system"] != "thermal":
        return None  # tens of thousands of unknowns: minutes in dense arithmetic
    # block tridiagonal by grid column (a diffusion matrix: its diagonal blocks are well conditioned)
    NX, NY = case["nx"] + 1, case["ny"] + 1
    new = lambda k: (k % NX) * NY + k // NX
    rows, cols = new(rows), new(cols)
    D = torch.zeros(3, NX, NY, NY, dtype=torch.float64, device="cuda")
    D[cols // NY - rows // NY + 1, rows // NY, rows % NY, cols % NY] = vals
    r = rhs.reshape(NY, NX).T.clone()
    up = torch.zeros(NX, NY, NY + 1, dtype=torch.float64, device="cuda")
    for i in range(NX):
        A, rr = D[1, i], r[i]
        if i:
            A, rr = A - D[0, i] @ up[i - 1, :, :NY], rr - D[0, i] @ up[i - 1, :, NY]
        up[i] = torch.linalg.solve(A, torch.cat([D[2, i], rr[:, None]], 1))
    u = torch.zeros(NX, NY, dtype=torch.float64, device="cuda")
    for i in range(NX - 1, -1, -1):
        u[i] = up[i, :, NY] - (up[i, :, :NY] @ u[i + 1] if i + 1 < NX else 0.0)
    return u.T.reshape(-1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "cycle" and case["box"] != "periodic":
        wl, P, grain = _box(case, seed)
        b = _Plain(wl, P.markers, grain)
        P.close()
        b.pre(wl.dt)
        b.post(wl.dt)
        b.thermal(wl.dt)
        b.pre(wl.dt)
        return {"nodal": b.nodal(NODAL_OUT), "residual": b.residual, "max_abs_sxx": b.max_abs_sxx, "max_T": b.max_T,
                "yielding": int(b.yielding)}
    if kind == "handover":
        wl, P, _ = _box(case, seed)
        b = _Plain(wl, P.markers)
        P.close()
        b.pre(wl.dt)
        b.post(wl.dt)
        b.thermal(wl.dt)
        whole = {"Mat": torch.int32, "cellX": torch.int32, "cellY": torch.int32}
        return {"markers": {f: b.m[f].to(whole.get(f, torch.float64)) for f in MARKER_OUT}, "nodal": b.nodal(NODAL_OUT),
                "residual": b.residual}
    if kind == "ensemble":
        out = []
        for wl in _members(case, seed):
            P = gpu.MicProblem(wl, capacity=wl.capacity)
            gpu.initialize_markers(P, *wl.nm, seed=wl.seed)
            b = _Plain(wl, P.markers)
            P.close()
            b.pre(wl.dt)
            out.append(b.nodal(("lastT", "etaN", "soxx", "soyy", "soxy")))
        return {"nodal": out}
    if kind == "solve":
        return _plain_solve(case, seed)
    return None  # a periodic box; a whole time step and a training run, whose every part feeds the next
