"""What a user of this framework has it do, as measurable cases.

A case is a dict of plain values; `prepare` makes what a program holds before
the call, `run` is one pass through the public entry points, `work` what a pass
cannot do without, and `exact` the same outputs in 64 bits from plain torch.

Kinds of case:
  cell       a periodic unit cell at normal incidence (slab, sphere or nanodisk
             scene), z-CPML, planar DFT flux sensors or none; a pass is `steps`
             time steps of a running simulation and the read of its flux
  spheres    one large grid in custom mode: CPML on six faces, many spheres, a
             point oscillator, optionally a box flux sensor
  batch      nanodisk cells of mixed sizes advanced together
  job        one complete small simulation: set-up, steps, sums and flux
  structure  voxelisation of a structure script into a material map
Simulations start from a running state (smooth random waves in all six field
components, made from the seed), so that every cell carries values."""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from aether_b200 import _abi as A
from aether_b200 import configs as CF
from aether_b200 import fdtd
from aether_b200 import lua_api

NM = 1e-9
C0, E0, MU0 = 299792458.0, 8.854187817e-12, 12.566370614e-7
ETA0 = math.sqrt(MU0 / E0)


def listed():
    return [
        # the smallest call: a test-sized dispersive column, where launches and latency are all of it
        {"name": "column_f64", "kind": "cell", "scene": "sphere", "precision": "f64", "nx": 12, "ny": 10, "nz": 90,
         "pml": 8, "radius": 3, "nl": 7, "steps": 64},
        # a dielectric slab with R/T flux at 61 wavelengths: the plain cell of every tutorial
        {"name": "slab_f64", "kind": "cell", "scene": "slab", "precision": "f64", "nx": 64, "ny": 64, "nz": 128,
         "pml": 16, "radius": 0, "nl": 61, "steps": 512},
        # the dispersive unit cell of the benchmark, in the reference's arithmetic
        {"name": "sphere_f64", "kind": "cell", "scene": "sphere", "precision": "f64", "nx": 128, "ny": 128, "nz": 256,
         "pml": 24, "radius": 16, "nl": 201, "steps": 256},
        # the same cell in single precision, as parameter sweeps run it
        {"name": "sphere_f32", "kind": "cell", "scene": "sphere", "precision": "f32", "nx": 128, "ny": 128, "nz": 256,
         "pml": 24, "radius": 16, "nl": 201, "steps": 256},
        # a cell whose sizes are odd and fit no tile, with a larger dispersive part
        {"name": "odd_f32", "kind": "cell", "scene": "sphere", "precision": "f32", "nx": 101, "ny": 77, "nz": 203,
         "pml": 17, "radius": 20, "nl": 33, "steps": 256},
        # one metasurface nanodisk cell alone: R/T sums only, no DFT planes
        {"name": "disk_f32", "kind": "cell", "scene": "disk", "precision": "f32", "nx": 60, "ny": 60, "nz": 200,
         "pml": 16, "radius": 18, "nl": 0, "steps": 512},
        # the same kind of cell at the largest period, in double precision
        {"name": "disk_f64", "kind": "cell", "scene": "disk", "precision": "f64", "nx": 120, "ny": 120, "nz": 200,
         "pml": 16, "radius": 40, "nl": 0, "steps": 256},
        # a scattering problem with a box flux sensor, six-sided CPML, double precision
        {"name": "spheres_f64", "kind": "spheres", "precision": "f64", "nx": 384, "ny": 384, "nz": 192, "pml": 32,
         "spheres": 60, "box": 64, "nl": 21, "steps": 32},
        # a large single grid in single precision, far beyond any cache
        {"name": "large_f32", "kind": "spheres", "precision": "f32", "nx": 768, "ny": 768, "nz": 384, "pml": 32,
         "spheres": 300, "box": 0, "nl": 0, "steps": 16},
        # a design sweep: nanodisk cells of periods 200-600 nm, stepped as one batch
        {"name": "batch_f32", "kind": "batch", "precision": "f32", "cells": 10, "nz": 200, "pml": 16, "mix": 5,
         "steps": 128},
        # a whole small simulation from host data: build, step, read the sums and the flux
        {"name": "job_f32", "kind": "job", "precision": "f32", "nx": 48, "nz": 200, "pml": 16, "nl": 101,
         "steps": 1024},
        # a structure script voxelised at the benchmark cell's resolution
        {"name": "structure", "kind": "structure", "nx": 160, "ny": 160, "nz": 240, "spheres": 40},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cell", "cell", "cell", "cell", "spheres", "batch", "job", "structure"])
    precision = rng.choice(["f64", "f32"])
    if kind == "cell":
        scene = rng.choice(["slab", "sphere", "disk"])
        nx, ny = _spread(rng, 10, 160), _spread(rng, 10, 160)
        pml = rng.randrange(8, 25)
        nz = _spread(rng, 2 * pml + 80, 256)
        nl = 0 if scene == "disk" else _spread(rng, 5, 201)
        radius = max(2, min(int(min(nx, ny) * rng.uniform(0.1, 0.4)), (int(0.7 * (nz - 2 * pml - 10)) - 20) // 2))
        cells = nx * ny * nz
        return {"kind": kind, "scene": scene, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "pml": pml,
                "radius": 0 if scene == "slab" else radius, "nl": nl,
                "steps": 64 * max(1, min(8, int(1e9 / cells / 64)))}
    if kind == "spheres":
        nx, ny, nz = _spread(rng, 72, 480), _spread(rng, 72, 480), _spread(rng, 72, 320)
        pml = rng.randrange(6, 29)
        box = rng.choice([0, min(nx, ny, nz) // 8])
        return {"kind": kind, "precision": precision, "nx": nx, "ny": ny, "nz": nz, "pml": pml,
                "spheres": _spread(rng, 8, 300), "box": box, "nl": _spread(rng, 3, 40) if box else 0,
                "steps": 8 * max(1, min(16, int(1e9 / (nx * ny * nz) / 8)))}
    if kind == "batch":
        return {"kind": kind, "precision": precision, "cells": rng.randrange(2, 11), "nz": _spread(rng, 120, 200),
                "pml": rng.randrange(8, 17), "mix": rng.randrange(1000), "steps": 64}
    if kind == "job":
        nx, nz = _spread(rng, 24, 100), _spread(rng, 120, 200)
        return {"kind": kind, "precision": precision, "nx": nx, "nz": nz, "pml": rng.randrange(8, 17),
                "nl": _spread(rng, 11, 201), "steps": 64 * max(2, min(16, int(1e9 / (nx * nx * nz) / 64)))}
    return {"kind": kind, "nx": _spread(rng, 32, 160), "ny": _spread(rng, 32, 160), "nz": _spread(rng, 32, 240),
            "spheres": _spread(rng, 4, 120)}


# ---- scenes ------------------------------------------------------------------

def _precision(case):
    return A.FP32 if case["precision"] == "f32" else A.FP64


def _cell_scene(case):
    nx, ny, nz, pml, nl = case["nx"], case["ny"], case["nz"], case["pml"], case["nl"]
    prec = _precision(case)
    if case["scene"] == "slab":
        return CF.slab_scene(nx=nx, ny=ny, nz_total=nz, pml=pml, slab=12, nl=nl, nsteps=20000, precision=prec)
    if case["scene"] == "sphere":
        return CF.sphere_scene(nx=nx, ny=ny, nz_total=nz, pml=pml, radius=case["radius"] * 2.5 * NM, nl=max(nl, 2),
                               nsteps=20000, sensor_gap=4, precision=prec)
    # nanodisk: a dispersive disk on a substrate, plane sums only
    nz_s = nz - 2 * pml - 10
    sub = int(round(0.35 * nz_s))
    m = np.zeros((nz_s, ny, nx), np.uint32)
    m[:sub] = 2
    x, y = np.arange(nx) - nx // 2, np.arange(ny) - ny // 2
    m[sub:sub + 8][:, (x[None, :] ** 2 + y[:, None] ** 2) <= case["radius"] ** 2] = 1
    g = A.grid_desc(nx, ny, nz_s, 5 * NM, mode=A.MODE_NORMAL, precision=prec, nt=20000, time_mod=0.5 / 0.99,
                    pml=(0, 0, 0, 0, pml, pml), pad=(0, 0, 0, 0, 5, 5), alpha=(0.05,) * 6)
    return CF.Scene(g, m, [CF.const_n(1.0), CF.gold_cp_model(), CF.const_n(1.45)], 20000,
                    normal=A.NormalDesc(1, 101, 400 * NM, 1000 * NM), name="disk")


def _spheres_scene(case):
    return CF.random_spheres_scene(n_total=(case["nx"], case["ny"], case["nz"]), pml=case["pml"],
                                   n_dielectric=case["spheres"], n_lorentz=max(1, case["spheres"] // 10),
                                   r_range=(20 * NM, 80 * NM), seed=case["spheres"], nsteps=5000,
                                   precision=_precision(case))


def _box(case, scene):
    """The box sensor around the centre: (box, nl, lambda_min, lambda_max)."""
    g, h = scene.grid, case["box"] // 2
    c = (g.nx // 2, g.ny // 2, g.nz // 2)
    return tuple(v for a in c for v in (a - h, a + h)), case["nl"], 450 * NM, 750 * NM


def _batch_scenes(case):
    rng = np.random.default_rng(case["mix"])
    return [CF.metasurface_cell(rng, nz_total=case["nz"], pml=case["pml"], precision=_precision(case), nsteps=20000,
                                flux_planes=False) for _ in range(case["cells"])]


def _job_scene(case, seed):
    period = case["nx"] * 5 * NM
    return CF.metasurface_cell(np.random.default_rng(seed), nz_total=case["nz"], pml=case["pml"], nl=case["nl"],
                               nsteps=case["steps"], period_range=(period, period), precision=_precision(case))


def _structure(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    d = 2.5 * NM
    size = (nx * d, ny * d, nz * d)

    def script(s):
        s.size(*size)
        s.add_layer("z", 0, 0.3 * size[2], 1)
        s.add_block(0.1 * size[0], 0.4 * size[0], 0.2 * size[1], 0.7 * size[1], 0.3 * size[2], 0.5 * size[2], 2)
        s.add_cylinder(0.6 * size[0], 0.5 * size[1], 0.3 * size[2], 0, 0, 0.2 * size[2], 0.15 * size[0], 3)
        for _ in range(case["spheres"]):
            x, y, z, r = rng.uniform(0, 1, 4)
            s.add_sphere(x * size[0], y * size[1], (0.5 + 0.5 * z) * size[2], (0.03 + 0.1 * r) * min(size), 4)
        s.loop(1, 1, 0)

    return script, (nx, ny, nz, d, d, d)


# ---- the running state -------------------------------------------------------

def _waves(shape, seed, comp, device, dtype):
    """One field component of a running simulation: three plane waves of 12 to
    40 cells per wavelength in random directions, E of order 1, H of order 1/eta0."""
    rng = np.random.default_rng([seed, comp])
    f = None
    for _ in range(3):
        k = rng.normal(size=3)
        k *= 2 * math.pi / rng.uniform(12, 40) / np.linalg.norm(k)
        phase, amp = rng.uniform(0, 2 * math.pi), rng.uniform(0.2, 1.0) / (1.0 if comp < 3 else ETA0)
        ax = [torch.arange(n, dtype=torch.float64, device=device) * float(kk) for n, kk in zip(shape, k[::-1])]
        # sin(a + b) from the one-dimensional sines, so that no large temporary is needed
        yx = ax[1][:, None] + ax[2][None, :] + phase
        part = torch.sin(ax[0])[:, None, None].to(dtype) * torch.cos(yx)[None].to(dtype)
        part += torch.cos(ax[0])[:, None, None].to(dtype) * torch.sin(yx)[None].to(dtype)
        f = part.mul_(amp) if f is None else f.add_(part, alpha=amp)
    return f


class _Array:
    """A device array of a simulation, for torch's zero-copy conversion; the
    tensor holds this object, and so the simulation, for as long as it lives."""

    def __init__(self, sim, ptr, shape, typestr):
        self.sim = sim
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


def _fields(sim):
    """Zero-copy tensors (nz, ny, nx) of Ex..Hz (aefdtd_field_device_ptr)."""
    d = sim.dims()
    out = []
    for c in range(6):
        p = ctypes.c_void_p()
        sim._c(sim._lib.aefdtd_field_device_ptr(sim._h, c, ctypes.byref(p)))
        kind = "<f4" if sim.grid.precision == A.FP32 else "<f8"
        out.append(torch.as_tensor(_Array(sim, p.value, (d.nz, d.ny, d.nx), kind), device="cuda"))
    return out


def _running(scene, seed):
    """The simulation of a scene with its fields set to a running state."""
    sim = fdtd.build_simulation(scene)
    sim.synchronize()
    fields = _fields(sim)
    for c, f in enumerate(fields):
        f.copy_(_waves(tuple(f.shape), seed, c, f.device, f.dtype))
    torch.cuda.synchronize()
    return sim, fields


def prepare(case, seed):
    kind = case["kind"]
    if kind == "structure":
        script, grid = _structure(case, seed)
        return {"case": case, "structure": lua_api.Structure(script), "grid": grid}
    if kind == "job":
        return {"case": case, "scene": _job_scene(case, seed)}
    if kind == "batch":
        sims, fields = [], []
        batch = fdtd.Batch()
        for i, scene in enumerate(_batch_scenes(case)):
            sim, f = _running(scene, seed + 1000 * i)
            batch.add(sim, 200000)
            sims.append(sim)
            fields.append(f)
        return {"case": case, "batch": batch, "sims": sims, "fields": fields}
    scene = _cell_scene(case) if kind == "cell" else _spheres_scene(case)
    if kind == "cell" and case["nl"] == 0:
        scene.sensors = []
    sim, fields = _running(scene, seed)
    boxes = []
    if kind == "spheres" and case["box"]:
        boxes.append(sim.add_box_sensor(*_box(case, scene)))
    return {"case": case, "sim": sim, "fields": fields, "boxes": boxes}


def _spectrum(case, values):
    """A single-precision run's spectra carry single precision."""
    return np.asarray(values, np.float32) if case["precision"] == "f32" else values


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "structure":
        return state["structure"].discretize(*state["grid"])
    if kind == "job":
        got = fdtd.run(state["scene"], want_fields=False)
        return {"sums": _spectrum(case, got["plane_sums"]), "flux": [_spectrum(case, f) for f in got["flux"]]}
    if kind == "batch":
        state["batch"].run(case["steps"])
        return {"fields": state["fields"]}
    sim = state["sim"]
    sim.step(case["steps"])
    sim.synchronize()
    out = {"fields": state["fields"]}
    if sim.sensor_nl:
        out["flux"] = [_spectrum(case, sim.sensor_flux(i)) for i in range(len(sim.sensor_nl))]
    if state["boxes"]:
        out["box"] = [_spectrum(case, sim.box_flux(b)) for b in state["boxes"]]
    return out


# ---- what a pass cannot do without ---------------------------------------------

def _scene_work(scene, planes, steps):
    """Per time step every field value and material id is read once and every
    new field value written once, with the CPML and pole state of the cells
    that have it; the DFT accumulators once per pass. 60 operations per cell
    and step, four per sample and wavelength."""
    g = scene.grid
    nx, ny, nz = scene.total_dims()
    s = 4 if g.precision == A.FP32 else 8
    cells = nx * ny * nz
    pml, _ = scene.padded_faces()
    psi = 4 * ((pml[0] + pml[1]) * ny * nz + nx * (pml[2] + pml[3]) * nz + nx * ny * (pml[4] + pml[5]))
    poles = sum(int((scene.map == i).sum()) * (m.n_debye + m.n_drude + m.n_lorentz + m.n_critpoint)
                for i, m in enumerate(scene.materials) if m.n_debye + m.n_drude + m.n_lorentz + m.n_critpoint)
    per_step = cells * (12 * s + (1 if len(scene.materials) <= 256 else 2)) + 2 * s * psi + 2 * 6 * s * poles
    samples = sum(6 * p * nl for p, nl in planes)
    return per_step * steps + 32 * samples, (60.0 * cells + 4.0 * samples) * steps


def work(case):
    kind = case["kind"]
    if kind == "structure":
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 4 * cells, "flops": 10.0 * cells * case["spheres"]}
    if kind == "batch":
        parts = [_scene_work(s, [], case["steps"]) for s in _batch_scenes(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind == "job":
        scene = _job_scene(case, 0)
        planes = [(case["nx"] ** 2, case["nl"])] * 2
    elif kind == "cell":
        scene = _cell_scene(case)
        planes = [(case["nx"] * case["ny"], case["nl"])] * (2 if case["nl"] else 0)
    else:
        scene = _spheres_scene(case)
        planes = [(case["box"] ** 2, case["nl"])] * (6 if case["box"] else 0)
    b, f = _scene_work(scene, planes, case["steps"])
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, in plain torch -----------------------------------------

def _poles(m):
    """(a, b) of each term a e^{bt} of a material, and its conductivity."""
    out, sigma = [], 0.0
    for n in range(m.n_debye):
        ds, t0 = m.debye[n][0], m.debye[n][1]
        out.append((ds / t0 + 0j, -1.0 / t0 + 0j))
    for n in range(m.n_drude):
        wd, g = m.drude[n][0], m.drude[n][1]
        out.append((-wd * wd / g + 0j, -g + 0j))
        sigma += E0 * wd * wd / g
    for n in range(m.n_lorentz):
        a, o, g = (m.lorentz[n][i] for i in range(3))
        beta = complex(o * o - g * g / 4) ** 0.5
        out.append((-1j * a * o * o / beta, -g / 2 + 1j * beta))
    for n in range(m.n_critpoint):
        a, o, p, g = (m.critpoint[n][i] for i in range(4))
        out.append((-2j * a * o * np.exp(-1j * p), -g + 1j * o))
    return out, sigma


class _Yee:
    """The time loop of one scene in 64 bits: Yee updates, CPML, recursive
    convolution, plane injection or oscillator, DFT planes and plane sums."""

    def __init__(self, scene, device):
        self.sc, g = scene, scene.grid
        self.dev, self.dt = device, scene.dt()
        self.n = scene.total_dims()[::-1]                     # nz, ny, nx
        self.D = (g.dz, g.dy, g.dx)
        self.t = 0
        pml, pad = scene.padded_faces()
        self.pml = [(pml[4], pml[5]), (pml[2], pml[3]), (pml[0], pml[1])]
        self.org = (pml[4] + pad[4], pml[2] + pad[2], pml[0] + pad[0])
        m = torch.from_numpy(scene.map.astype(np.int64)).to(device)
        for ax, (lo, n) in enumerate(zip(self.org, self.n)):  # edges replicated into pads and PML
            idx = (torch.arange(n, device=device) - lo).clamp(0, m.shape[ax] - 1)
            m = m.index_select(ax, idx)
        self.map = m
        dt = self.dt
        c1, c3, ce, self.disp = [], [], [], []
        for i, mat in enumerate(scene.materials):
            poles, sigma = _poles(mat)
            eff = mat.eps_inf + sigma * dt / E0
            eff += sum((a / b * (np.exp(b * dt) - 1)).real for a, b in poles)
            c1.append(mat.eps_inf / eff if poles else 1.0)
            c3.append(1.0 / eff if poles else 0.0)
            ce.append(dt / (E0 * eff))
            where = (m == i).nonzero(as_tuple=True) if poles else ()
            if poles and where[0].numel():
                rec = torch.tensor([np.exp(b * dt) for a, b in poles], dtype=torch.complex128, device=device)
                chi = torch.tensor([-a / b * (1 - np.exp(b * dt)) ** 2 for a, b in poles], dtype=torch.complex128,
                                   device=device)
                psi = torch.zeros((3, len(poles), where[0].numel()), dtype=torch.complex128, device=device)
                self.disp.append((where, rec[:, None], chi[:, None], psi, c3[-1]))
        as_t = lambda v: torch.tensor(v, dtype=torch.float64, device=device)  # noqa: E731
        self.c1 = as_t(c1)[m] if self.disp else None
        self.ce = as_t(ce)[m]
        self.f = [torch.zeros(self.n, dtype=torch.float64, device=device) for _ in range(6)]
        self.tab, self.psi = {}, {}
        for ax in range(3):
            lo, hi = self.pml[ax]
            if not lo and not hi:
                continue
            n, face = self.n[ax], (4, 2, 0)[ax]
            for half in (0, 1):
                b, c, ik = np.zeros(n), np.zeros(n), np.ones(n)
                for i in range(n):
                    at = i + 0.5 * half
                    x, f = ((lo - at) / lo, face) if at < lo else ((at - n + hi) / hi, face + 1) if at > n - hi else (0, 0)
                    if x <= 0:
                        continue
                    sig = 0.8 * 5 / (ETA0 * self.D[ax]) * g.pml_sigma[f] * x ** 4
                    alp, kap = g.pml_alpha[f] * (1 - x) ** 2, 1 + (g.pml_kappa[f] - 1) * x ** 4
                    ik[i] = 1 / kap
                    if (half == 0 and (1 <= i < lo or i >= n - hi + 1)) or (half and (i < lo or n - hi <= i < n - 1)):
                        b[i] = math.exp(-(sig / kap + alp) * dt / E0)
                        c[i] = sig / (sig * kap + kap * kap * alp) * (b[i] - 1) / self.D[ax]
                shape = [1, 1, 1]
                shape[ax] = n
                self.tab[half, ax] = tuple(as_t(v).reshape(shape) for v in (b, c, ik))
        self._source()
        self.dft = []
        for s in scene.sensors:
            self.add_plane(s.orientation, list(s.box), s.nl, s.lambda_min, s.lambda_max)

    def _source(self):
        sc, dt = self.sc, self.dt
        self.osc = []
        for s in sc.sources:
            w1, w2 = 2 * math.pi * C0 / s.lambda_max, 2 * math.pi * C0 / s.lambda_min
            dw = abs(w2 - w1) / (2 * math.sqrt(-math.log(math.sqrt(0.1))))
            shift = int(math.sqrt(-4 / (dw * dw) * math.log(1e-7)) / dt)
            b = [s.box[i] + self.org[2 - i // 2] for i in range(6)]
            self.osc.append(((0, 0, 1, 1, 2, 2)[s.orientation], b, (w1 + w2) / 2, dw, shift))
        self.sums = []
        if sc.normal is None:
            return
        nd, dz = sc.normal, self.D[0]
        self.top, self.bottom = self.org[0] + sc.grid.nz, self.org[0]
        n_sup = math.sqrt(sc.materials[int(self.map[self.top, 0, 0])].eps_inf)
        wi, wf = 2 * math.pi * C0 / nd.lambda_min, 2 * math.pi * C0 / nd.lambda_max
        om = (wi + wf) / 2
        k, width = om / C0 * n_sup, 2 * C0 / abs(0.5 * (wi - om)) / n_sup
        start = (self.top - 1) * dz
        c1 = start + width * math.sqrt(-math.log(1e-4))

        def pulse(z, t):
            b = (-z - C0 * t / n_sup + c1) / width
            return math.exp(-b * b) * math.cos(-k * z - om * t)

        tm = nd.polarization == 1
        h0 = n_sup / (C0 * MU0)
        self.eps_sup, self.pulse = n_sup * n_sup, pulse
        self.amp = {"ex": float(tm), "ey": float(not tm), "hx": h0 * (not tm), "hy": -h0 * tm}

    def add_plane(self, orientation, box, nl, lmin, lmax):
        lo = [max(0, min(box[2 * i] + self.org[2 - i], self.n[2 - i])) for i in range(3)]
        hi = [max(0, min(box[2 * i + 1] + self.org[2 - i], self.n[2 - i])) for i in range(3)]
        ax = orientation // 2                                 # 0 x, 1 y, 2 z
        hi[ax] = lo[ax] + 1
        at = tuple(torch.arange(lo[2 - i], hi[2 - i], device=self.dev) for i in range(3))
        w = 2 * math.pi * C0 / np.linspace(lmin, lmax, nl)
        acc = torch.zeros((6, nl, math.prod(len(a) for a in at)), dtype=torch.complex128, device=self.dev)
        self.dft.append({"ax": ax, "sign": 1 - 2 * (orientation % 2), "at": at,
                         "w": torch.tensor(w, dtype=torch.float64, device=self.dev), "acc": acc,
                         "area": self.D[0] * self.D[1] * self.D[2] / self.D[2 - ax]})

    def _diff(self, c, ax, half):
        """Backward (E side) or forward (H side) difference along ax, periodic."""
        f = self.f[c]
        return torch.roll(f, -1, ax).sub_(f) if half else f - torch.roll(f, 1, ax)

    def _curl(self, half, target, comp, sign, ax, out):
        """out += sign (d comp / d ax, with the CPML's stretch and memory)."""
        d = self._diff(comp, ax, half)
        if (half, ax) not in self.tab:
            return out.add_(d, alpha=sign / self.D[ax])
        b, c, ik = self.tab[half, ax]
        p = self.psi.get((target, ax))
        p = c * d if p is None else p.mul_(b).add_(c * d)
        self.psi[target, ax] = p
        return out.add_(d * ik, alpha=sign / self.D[ax]).add_(p, alpha=sign)

    def _pec(self, half):
        """Conducting planes behind the CPML, at the first E and the last H
        index. A component's two axes are finished one after the other, so a
        plane of its first axis keeps the second axis' CPML memory term."""
        for comp, first, second, sign in ((0, 1, 0, -1), (1, 2, 0, 1), (2, 2, 1, -1)):
            f, scale = self.f[comp + 3 * half], self.dt / MU0 if half else self.ce
            if any(self.pml[first]):
                at = self.n[first] - 1 if half else 0
                kept = self.psi.get((comp + 3 * half, second))
                if kept is None:
                    f.select(first, at).zero_()
                else:
                    factor = scale if half else scale.select(first, at)
                    f.select(first, at).copy_(kept.select(first, at) * factor * (-sign if half else sign))
            if any(self.pml[second]):
                f.select(second, self.n[second] - 1 if half else 0).zero_()

    def step(self):
        t, dt, f = self.t, self.dt, self.f
        old = [[f[c][where] for c in range(3)] for where, *_ in self.disp]
        # (target, first: +d comp / d axis, second: -d comp / d axis); axes 0 z, 1 y, 2 x
        for e, (a, ax_a), (b, ax_b) in ((0, (5, 1), (4, 0)), (1, (3, 0), (5, 2)), (2, (4, 2), (3, 1))):
            out = torch.zeros_like(f[e])
            self._curl(0, e, a, 1.0, ax_a, out)
            self._curl(0, e, b, -1.0, ax_b, out)
            out.mul_(self.ce)
            if self.c1 is not None:
                f[e].mul_(self.c1)
            f[e].add_(out)
        for (where, rec, chi, psi, c3), ev in zip(self.disp, old):
            for c in range(3):
                psi[c].mul_(rec).add_(chi * ev[c][None])
                f[c][where] += c3 * psi[c].real.sum(0)
        self._pec(0)
        if self.sc.normal is not None:
            z, k = self.top - 1, self.D[0]
            f[0][z] -= dt / (k * E0) / self.eps_sup * self.amp["hy"] * self.pulse((z + 0.5) * k, t * dt)
            f[1][z] += dt / (k * E0) / self.eps_sup * self.amp["hx"] * self.pulse((z + 0.5) * k, t * dt)
        for comp, b, w0, dw, shift in self.osc:
            v = math.cos(w0 * t * dt) * math.exp(-(dw / 2 * (t - shift) * dt) ** 2) * 50
            f[comp][b[4]:b[5], b[2]:b[3], b[0]:b[1]] += v
        for h, (a, ax_a), (b, ax_b) in ((3, (1, 0), (2, 1)), (4, (2, 2), (0, 0)), (5, (0, 1), (1, 2))):
            out = torch.zeros_like(f[h])
            self._curl(1, h, a, 1.0, ax_a, out)
            self._curl(1, h, b, -1.0, ax_b, out)
            f[h].add_(out, alpha=dt / MU0)
        self._pec(1)
        if self.sc.normal is not None:
            z, k = self.top - 1, self.D[0]
            f[3][z] += dt / (k * MU0) * self.amp["ey"] * self.pulse(z * k, (t + 0.5) * dt)
            f[4][z] -= dt / (k * MU0) * self.amp["ex"] * self.pulse(z * k, (t + 0.5) * dt)
            self._plane_sums()
        for s in self.dft:
            self._sample(s)
        self.t += 1

    def _plane_sums(self):
        dz, tb, cells = self.D[0], (self.t + 0.5) * self.dt, self.n[1] * self.n[2]
        amp = (self.amp["ex"], self.amp["ey"], 0.0)
        zr, zt = self.top - 2, self.bottom
        inc = [[a * self.pulse(z * dz, tb) for a in amp] for z in (zr, zt)]
        r = [self.f[c][zr].sum() - cells * inc[0][c] for c in range(3)]
        tr = [self.f[c][zt].sum() for c in range(3)]
        as_t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.sums.append(torch.stack([as_t(v) for v in ([cells * x for x in inc[0]] + r + [cells * x for x in inc[1]] + tr)]))

    def _sample(self, s):
        f, n = self.f, self.n
        z, y, x = s["at"]
        up = [(a + 1) % m for a, m in zip(s["at"], n)]

        def at(c, zi, yi, xi):
            return f[c][zi[:, None, None], yi[None, :, None], xi[None, None, :]]

        e = [(at(0, z, y, x) + at(0, z, up[1], x) + at(0, up[0], y, x) + at(0, up[0], up[1], x)) / 4,
             (at(1, z, y, x) + at(1, z, y, up[2]) + at(1, up[0], y, x) + at(1, up[0], y, up[2])) / 4,
             (at(2, z, y, x) + at(2, z, y, up[2]) + at(2, z, up[1], x) + at(2, z, up[1], up[2])) / 4]
        h = [(at(3, z, y, x) + at(3, z, y, up[2])) / 2, (at(4, z, y, x) + at(4, z, up[1], x)) / 2,
             (at(5, z, y, x) + at(5, up[0], y, x)) / 2]
        for c in range(6):
            ph = torch.exp(1j * s["w"] * ((self.t + (0.5 if c > 2 else 0.0)) * self.dt))
            s["acc"][c] += ph[:, None] * (e + h)[c].reshape(1, -1)

    def flux(self, s):
        a, (u, v) = s["acc"], ((1, 2), (2, 0), (0, 1))[s["ax"]]
        return s["sign"] * s["area"] * (a[u] * a[3 + v].conj() - a[v] * a[3 + u].conj()).real.sum(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "structure":
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "job":
        y = _Yee(_job_scene(case, seed), dev)
        for _ in range(case["steps"]):
            y.step()
        return {"sums": torch.stack(y.sums, 1), "flux": [y.flux(s) for s in y.dft]}
    dtype = torch.float32 if case["precision"] == "f32" else torch.float64
    if kind == "batch":
        scenes = _batch_scenes(case)
    else:
        scenes = [_cell_scene(case) if kind == "cell" else _spheres_scene(case)]
        if kind == "cell" and case["nl"] == 0:
            scenes[0].sensors = []
    fields = []
    for i, scene in enumerate(scenes):
        y = _Yee(scene, dev)
        for c in range(6):
            y.f[c].copy_(_waves(tuple(y.n), seed + 1000 * i, c, dev, dtype))
        if kind == "spheres" and case["box"]:
            (x1, x2, y1, y2, z1, z2), nl, lmin, lmax = _box(case, scene)
            for o, b in ((1, (x1, x1 + 1, y1, y2, z1, z2)), (0, (x2 - 1, x2, y1, y2, z1, z2)),
                         (3, (x1, x2, y1, y1 + 1, z1, z2)), (2, (x1, x2, y2 - 1, y2, z1, z2)),
                         (5, (x1, x2, y1, y2, z1, z1 + 1)), (4, (x1, x2, y1, y2, z2 - 1, z2))):
                y.add_plane(o, b, nl, lmin, lmax)
        for _ in range(case["steps"]):
            y.step()
        fields.append(y.f)
    if kind == "batch":
        return {"fields": fields}
    out = {"fields": fields[0]}
    if kind == "cell" and y.dft:
        out["flux"] = [y.flux(s) for s in y.dft]
    if kind == "spheres" and case["box"]:
        out["box"] = [sum(y.flux(s) for s in y.dft)]
    return out
