"""The work users of the engine have it do, as measurable cases.

A case is one program's inner loop over the public entry points: flow steps followed by a device
read of the macroscopic fields, single steps under a monitor, a geometry set from a surface, the
gray-lattice forward and reverse sweeps under torch.autograd, and a coupled multiphysics cycle.

listed()  the cases that are watched; draw() gives more of the same ranges: lattices of 24^3 cells
          up to 16.7 M cells (the listed ones reach 512^3), odd and even rows, both lattices, every
          storage, both collisions, with and without Smagorinsky, walls, forces and gray cells.
prepare() the solver with its geometry and initial state, as a program holds it before the loop.
run()     one pass; the outputs are the macroscopic fields, the populations (the handle's own
          buffer) and whatever else the pass computes.
exact()   the macroscopic fields, gradients and scalars in 64 bits, from a plain torch lattice
          Boltzmann method in its logical (two-lattice) form, and a ray-cast voxelizer.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import cfd_solvers_b200 as cs
from cfd_solvers_b200 import bindings
from cfd_solvers_b200.autograd import device_fields, gray_lbm
from cfd_solvers_b200.geometry import icosphere, transform_surface
from cfd_solvers_b200.multiphysics import (ParticleVector3, ResidentFlowDiagnostics3D, ResidentFreeSurface3D,
                                           ResidentParticles3D, ResidentThermalD3Q7)

DEVICE = "cuda"

_FLOW = {"kind": "flow", "lattice": "d3q19", "storage": "fp32", "collision": "trt", "les": False, "geometry": "periodic",
         "tau": 0.6, "force": 0.0, "rounding": "stochastic"}


def _flow(**kw):
    return dict(_FLOW, **kw)


def listed():
    return [
        # Small validation runs are periodic Taylor-Green boxes, stepped in long calls: launches and gaps count.
        _flow(name="taylor_green_64", nx=64, ny=64, nz=64, steps=100, collision="bgk"),
        # A monitored run: one step per call with the conservation sums read after each, on a small cavity.
        _flow(name="monitored_cavity_32", kind="monitored", nx=32, ny=32, nz=32, steps=16, geometry="cavity", les=True,
              tau=0.51),
        # The headline workload: lid-driven cavity, TRT + Smagorinsky, FP32.
        _flow(name="cavity_512", nx=512, ny=512, nz=512, steps=10, geometry="cavity", les=True, tau=0.51),
        # The same physics in shifted FP16 storage at an everyday size.
        _flow(name="cavity_256_fp16", nx=256, ny=256, nz=256, steps=20, geometry="cavity", les=True, tau=0.51,
              storage="fp16s"),
        # Porous channel flow in FP16: bounce-back on many curved surfaces, body force.
        _flow(name="spheres_512x256x256_fp16", nx=512, ny=256, nz=256, steps=10, geometry="spheres", force=1e-6,
              storage="fp16s"),
        # Porous channel of odd extents in FP32.
        _flow(name="spheres_301x155x133", nx=301, ny=155, nz=133, steps=20, geometry="spheres", force=1e-6,
              collision="bgk"),
        # D3Q27 in FP16: turbulence runs on the larger stencil.
        _flow(name="cavity_d3q27_256_fp16", lattice="d3q27", nx=256, ny=256, nz=256, steps=10, geometry="cavity",
              les=True, tau=0.51, storage="fp16s"),
        # FP64 convergence studies on a periodic box.
        _flow(name="taylor_green_fp64_128", nx=128, ny=128, nz=128, steps=20, collision="bgk", storage="fp64"),
        # Sensitivities of a gray channel (topology optimisation): forward and reverse sweep, FP32.
        _flow(name="gray_adjoint_128", kind="adjoint", nx=128, ny=128, nz=128, steps=96, interval=64,
              geometry="channel", force=1e-6),
        # The same on D3Q27 with FP16 frames, where checkpoints are large.
        _flow(name="gray_adjoint_d3q27_160_fp16", kind="adjoint", lattice="d3q27", nx=160, ny=160, nz=160, steps=32,
              interval=16, geometry="channel", force=1e-6, storage="fp16s"),
        # A new geometry: a triangulated body set into a channel, initialised and started.
        _flow(name="body_256x128x128", kind="body", nx=256, ny=128, nz=128, steps=10, subdivisions=4, tau=0.55,
              les=True),
        # Coupled cycle: buoyant heat, free surface, two-way particles and Q on the flow's device views.
        _flow(name="coupled_192", kind="coupled", nx=192, ny=192, nz=192, steps=4, particles=1 << 18, tau=0.55),
    ]


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        dims = [_extent(rng, 24, 400) for _ in range(3)]
        if rng.random() < 0.5:
            dims[0] += dims[0] % 2  # rows of even length are as common as all others together
        cells = dims[0] * dims[1] * dims[2]
        if cells <= 1 << 24:
            break
    c = _flow(nx=dims[0], ny=dims[1], nz=dims[2])
    kind = rng.choice(["flow"] * 5 + ["monitored", "adjoint", "body", "coupled"])
    steps = max(4, min(100, (1 << 28) // cells))
    c["kind"] = kind
    c["lattice"] = rng.choice(["d3q19", "d3q19", "d3q27"])
    c["collision"] = rng.choice(["bgk", "trt"])
    c["tau"] = round(rng.uniform(0.53, 0.8), 3)
    c["storage"] = rng.choice(["fp32", "fp32", "fp16s", "fp16s", "fp64"])
    c["rounding"] = rng.choice(["stochastic", "nearest"])
    if kind in ("flow", "monitored"):
        c["les"] = rng.random() < 0.5
        c["geometry"] = rng.choice(["periodic", "cavity", "spheres", "channel"])
        c["force"] = 1e-6 if c["geometry"] in ("spheres", "channel") else 0.0
        c["steps"] = steps if kind == "flow" else min(steps, 16)
    elif kind == "adjoint":
        for k in ("nx", "ny", "nz"):  # the checkpoints of a reverse sweep hold many lattices
            c[k] = (c[k] + 1) // 2
        c["geometry"], c["force"] = rng.choice(["periodic", "channel"]), 1e-6
        c["steps"], c["interval"] = min(max(8, steps), 64), rng.choice([8, 16, 64])
    elif kind == "body":
        c["les"], c["steps"], c["subdivisions"] = rng.random() < 0.5, min(steps, 20), rng.choice([2, 3, 4])
    else:
        c["storage"] = rng.choice(["fp32", "fp16s"])
        c["steps"], c["particles"] = min(steps, 8), 1 << rng.randrange(10, 19)
    return c


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _flags(case, seed):
    """Cell flags (uint8, [nz][ny][nx]) of the case's geometry, or None."""
    g, nx, ny, nz = case["geometry"], case["nx"], case["ny"], case["nz"]
    if g == "periodic":
        return None
    f = torch.zeros((nz, ny, nx), dtype=torch.uint8, device=DEVICE)
    if g == "cavity":
        f[:, :, 0] = f[:, :, -1] = 1
        f[:, 0, :] = 1
        f[0] = f[-1] = 1
        f[:, -1, :] = 2
        return f
    f[:, 0, :] = f[:, -1, :] = 1
    f[0] = f[-1] = 1
    if g == "spheres":  # random solid spheres, about a tenth of the volume
        rng = np.random.default_rng(int(seed))
        rmax = min(12.0, 0.2 * min(nx, ny, nz))
        rmin = rmax / 3.0
        count = max(1, int(0.1 * nx * ny * nz / (math.pi / 3.0 * (rmax ** 4 - rmin ** 4) / (rmax - rmin))))
        ax = [torch.arange(e, device=DEVICE, dtype=torch.float32) + 0.5 for e in (nx, ny, nz)]
        for _ in range(count):
            r = rng.uniform(rmin, rmax)
            c = [rng.uniform(0, e) for e in (nx, ny, nz)]
            (x0, x1), (y0, y1), (z0, z1) = [(max(0, int(p - r) - 1), min(e, int(p + r) + 2))
                                            for p, e in zip(c, (nx, ny, nz))]
            d2 = ((ax[0][x0:x1] - c[0]) ** 2)[None, None, :] + ((ax[1][y0:y1] - c[1]) ** 2)[None, :, None]
            d2 = d2 + ((ax[2][z0:z1] - c[2]) ** 2)[:, None, None]
            f[z0:z1, y0:y1, x0:x1] |= (d2 <= r * r).to(torch.uint8)
    return f


def _fields(case, seed, amplitude=0.04):
    """rho | ux | uy | uz (float32, [4][nz][ny][nx]): divergence-free shear modes with random phases."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(int(seed) + 77)
    wave = []
    for e in (nx, ny, nz):
        x = (torch.arange(e, device=DEVICE, dtype=torch.float64) + 0.5) / e
        wave.append([torch.sin(2 * math.pi * (k * x + rng.uniform())) for k in (1, 2, 1, 2)])
    wx, wy, wz = wave
    out = torch.empty((4, nz, ny, nx), dtype=torch.float32, device=DEVICE)
    out[0] = 1.0
    amp = amplitude * rng.uniform(0.5, 1.0, 3)
    out[1] = (amp[0] * wy[0][None, :] * wz[1][:, None]).float()[:, :, None]
    out[2] = (amp[1] * wx[0][None, :] * wz[0][:, None]).float()[:, None, :]
    out[3] = (amp[2] * wx[1][None, :] * wy[2][:, None]).float()[None, :, :]
    return out


def _lid(seed):
    return float(np.float32(0.05 + 0.05 * np.random.default_rng(int(seed) + 5).uniform()))


def _gray(case, seed):
    n = case["nx"] * case["ny"] * case["nz"]
    return 0.2 * torch.rand(n, device=DEVICE, generator=_generator(seed + 3))


def _body(case, seed):
    """A closed sphere of unit-box coordinates, rotated and shifted."""
    rng = np.random.default_rng(int(seed) + 11)
    s = icosphere((0.0, 0.0, 0.0), 0.2, case["subdivisions"])
    return transform_surface(s, 0.5 + 0.1 * rng.uniform(-1, 1, 3), rng.uniform(-1, 1, 3), rng.uniform(0, 3))


def _particles(case, seed):
    rng = np.random.default_rng(int(seed) + 21)
    rec = np.zeros((case["particles"], 8))
    rec[:, :3] = rng.uniform(0, 1, (case["particles"], 3)) * (case["nx"], case["ny"], case["nz"])
    rec[:, 6], rec[:, 7] = 1e-4, 20.0
    return rec


def _temperature(case, seed):
    w = _fields(case, seed + 31, 1.0)
    return (300.0 + w[1] + w[2]).reshape(-1).cpu().numpy()


class _View:
    """A device buffer of a handle, for torch.as_tensor; keeps its owner alive."""

    def __init__(self, owner, pointer, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (int(pointer), False),
                                         "version": 3, "strides": None}


def _view(owner, pointer, shape, typestr):
    return torch.as_tensor(_View(owner, pointer, shape, typestr), device=DEVICE)


def _init_fields(solver, fields):
    torch.cuda.current_stream().synchronize()
    solver.library.call("cfdx_lbm_init_fields", solver.handle, ctypes.c_void_p(fields.data_ptr()), bindings.DEVICE)


def prepare(case, seed):
    c = case
    s = cs.EsotericPullCudaSolver(cs.InPlaceLbmConfig(
        nx=c["nx"], ny=c["ny"], nz=c["nz"], tau=c["tau"], acceleration_x=c["force"], smagorinsky_les=c["les"],
        smagorinsky_cs=0.1 if c["les"] else 0.0, lattice=c["lattice"], collision=c["collision"], storage=c["storage"],
        fp16_rounding=c["rounding"], rounding_seed=int(seed) & 0xffff))
    state = {"case": c, "solver": s, "fields": _fields(c, seed)}
    flags = _flags(c, seed)
    if flags is not None:
        s.set_flags(flags.reshape(-1))
        if c["geometry"] == "cavity":
            s.set_wall_velocity(2, _lid(seed), 0.0, 0.0)
    ptr, size = s.raw_populations()
    kind = {"fp32": "<f4", "fp16s": "<f2", "fp64": "<f8"}[c["storage"]]
    state["f"] = _view(s, ptr, (s.config.q, s.cells()), kind)
    if c["kind"] == "adjoint":
        state["ns"] = _gray(c, seed).requires_grad_()
        state["tau"] = torch.tensor(c["tau"], dtype=torch.float64, device=DEVICE, requires_grad=True)
        state["goal"] = state["fields"][1:].reshape(3, -1).clone()
        return state
    _init_fields(s, state["fields"])
    if c["kind"] == "body":
        state["body"] = _body(c, seed)
        channel = _flags(dict(c, geometry="channel"), seed).reshape(-1)
        state["channel"] = channel
    if c["kind"] == "coupled":
        th, fs = ResidentThermalD3Q7(s, 0.02), ResidentFreeSurface3D(s)
        pt, dg = ResidentParticles3D(s, c["particles"]), ResidentFlowDiagnostics3D(s)
        th.initialize_field(_temperature(c, seed))
        fs.initialize_half_space_x(c["nx"] / 2 + 0.25)
        pt.upload(_particles(c, seed))
        state.update(th=th, fs=fs, pt=pt, dg=dg)
        n = s.cells()
        own = (s, th, fs, pt, dg)
        state["fill"] = _view(own, fs.fill_device(), (n,), "<f4")
        state["points"] = _view(own, pt.device_state(), (8, c["particles"]), "<f4")
        state["q"] = _view(own, dg.q_criterion(s.refresh_device_macroscopic()), (n,), "<f4")
        state["t"] = _view(own, th.refresh_device_scalar(), (n,), "<f4")
    s.wait()
    return state


def run(state):
    c, s = state["case"], state["solver"]
    kind = c["kind"]
    out = {}
    if kind == "flow":
        s.step(c["steps"])
    elif kind == "monitored":
        for _ in range(c["steps"]):
            s.step(1)
            sums = s.reduce()
        out["sums"] = [sums["mass"], sums["kinetic_energy"], sums["max_speed"]]
    elif kind == "body":
        s.set_solid_surface(state["body"], base_flags=state["channel"])
        _init_fields(s, state["fields"])
        s.step(c["steps"])
    elif kind == "adjoint":
        rho, u = gray_lbm(state["ns"], state["tau"], s, c["steps"], c["interval"],
                          lambda solver: _init_fields(solver, state["fields"]))
        grad_ns, grad_tau = torch.autograd.grad((u * state["goal"]).sum(), (state["ns"], state["tau"]))
        return {"rho": rho.detach(), "u": u.detach(), "grad_ns": grad_ns, "grad_tau": grad_tau}
    else:
        th, fs, pt, dg = state["th"], state["fs"], state["pt"], state["dg"]
        for _ in range(c["steps"]):
            flow = s.refresh_device_macroscopic()
            force = s.device_local_acceleration(clear=True)
            th.step(flow, 1)
            th.add_boussinesq_acceleration(force, 300.0, 1e-4, ParticleVector3(0.0, -1.0, 0.0))
            fs.advect(flow, 0.5)
            fs.add_surface_tension_acceleration(force, 1e-4)
            pt.advance(flow, force, 0.5, True)
            s.step(1)
        dg.q_criterion(s.refresh_device_macroscopic())
        th.refresh_device_scalar()
        out = {"fill": state["fill"], "points": state["points"], "q": state["q"], "t": state["t"]}
    rho, u = device_fields(s, torch.device(DEVICE, torch.cuda.current_device()))
    out.update(rho=rho, u=u, f=state["f"])
    return out


# -------------------------------------------------------------------- work
def work(case):
    """Bytes of every population read and written once per step (the state of a step is the input of the
    next), plus the fields the pass reads and writes; arithmetic of the collision at about 12 operations
    per population."""
    c = case
    n = c["nx"] * c["ny"] * c["nz"]
    q = 19 if c["lattice"] == "d3q19" else 27
    size = {"fp32": 4, "fp16s": 2, "fp64": 8}[c["storage"]]
    walls = 0 if c["geometry"] == "periodic" and c["kind"] != "body" else 1
    step = 2 * q * size + walls
    read = q * size + walls + 4 * (8 if c["storage"] == "fp64" else 4)
    steps, total = c["steps"], 0
    if c["kind"] == "adjoint":
        lam = 8 if c["storage"] == "fp64" else 4
        # forward; reverse: the state of the step read, the adjoint read and written, n_s, the gradient
        total = steps * (step + 4) + steps * (q * size + 2 * q * lam + 4 + walls) + read + 12 + 8
        flops = steps * n * q * 36.0
    else:
        total = steps * step + read
        flops = steps * n * q * 12.0
        if c["kind"] == "monitored":
            total += steps * (q * size + walls)
        elif c["kind"] == "body":
            total += 16 + q * size + 2
        elif c["kind"] == "coupled":
            # velocity out and in, acceleration out and in, temperature populations, fill; Q and T at the end
            total += steps * (q * size + 16 + 12 + 12 + 12 + 56 + 8) + q * size + 16 + 4 + 32
    return {"bytes": float(n) * total + 64.0 * c.get("particles", 0) * steps, "flops": flops}


def tolerance(case):
    """About four times the distance of the path from exact() (adjoint and coupled outputs hold small
    differences of the state: u under a weak force, gradients, the Q-criterion)."""
    if case["storage"] == "fp64":
        return {"rel": 1e-11, "max": 1e-9}
    if case["storage"] == "fp16s":  # the random bits of the stores move every population by about 2^-11
        return {"rel": 2e-2, "max": 0.8} if case["kind"] == "coupled" else {"rel": 6e-3, "max": 0.24}
    rel = {"adjoint": 2.5e-3, "coupled": 6e-4}.get(case["kind"], 2e-5)
    return {"rel": rel, "max": 40 * rel}


# ------------------------------------------------------------------- exact
_C = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
               (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1),
               (0, 1, -1), (0, -1, 1), (1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1),
               (1, -1, -1), (-1, 1, 1)])


def _weights(q):
    by = {19: (1 / 3, 1 / 18, 1 / 36), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}[q]
    return [by[int(np.abs(_C[i]).sum())] for i in range(q)]


def _opp(i):
    return 0 if i == 0 else (i + 1 if i % 2 else i - 1)


def _f32(v):
    return float(np.float32(v))


def _dot(i, v):
    t = None
    for a in range(3):
        if _C[i][a]:
            x = v[a] if _C[i][a] > 0 else -v[a]
            t = x if t is None else t + x
    return t


def _shift(a, c):
    """The value each cell receives from its upstream neighbour n - c (periodic)."""
    d = [k for k in range(3) if c[k]]
    return torch.roll(a, [int(c[k]) for k in d], [2 - k for k in d]) if d else a


def _equilibrium(rho, u, q):
    w = _weights(q)
    sq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    out = [w[0] * rho * (1 - sq)]
    for i in range(1, q):
        cu = _dot(i, u)
        out.append(w[i] * rho * (1 + 3 * cu + 4.5 * cu * cu - sq))
    return out


def _moments(x, q):
    rho = sum(x[1:], x[0])
    j = []
    for a in range(3):
        t = None
        for i in range(1, q):
            if _C[i][a]:
                v = x[i] if _C[i][a] > 0 else -x[i]
                t = v if t is None else t + v
        j.append(t)
    return rho, [v / rho for v in j]


def _collide(c, x, tau, accel, ns):
    """Post-collision populations: TRT or BGK with Guo forcing, Smagorinsky and gray bounce-back."""
    q, w = len(x), _weights(len(x))
    rho, u = _moments(x, q)
    if accel is not None:
        u = [v + 0.5 * a for v, a in zip(u, accel)]
    if c["les"]:
        k, total = 18.0 * math.sqrt(2.0) * _f32(0.1) ** 2, 0.0
        for a in range(3):
            for b in range(a, 3):
                p = -rho * (u[a] * u[b] + (1 / 3 if a == b else 0.0))
                for i in range(q):
                    if _C[i][a] * _C[i][b]:
                        p = p + x[i] * int(_C[i][a] * _C[i][b])
                total = total + (1.0 if a == b else 2.0) * p * p
        tau = 0.5 * (tau + torch.sqrt(tau * tau + k * torch.sqrt(total) / rho))
    wp = 1.0 / tau
    wm = wp if c["collision"] == "bgk" else 1.0 / (0.5 + (3.0 / 16.0) / (tau - 0.5))
    sq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    uf = 0.0
    if accel is not None:
        f = [rho * a for a in accel]
        uf = u[0] * f[0] + u[1] * f[1] + u[2] * f[2]
    o0 = x[0] - wp * (x[0] - w[0] * rho * (1 - sq)) - (1 - 0.5 * wp) * w[0] * 3 * uf
    out = [None] * q
    out[0] = o0 if ns is None else (1 - ns) * o0 + ns * x[0]
    for i in range(1, q, 2):
        j = i + 1
        s, d, cu = x[i] + x[j], x[i] - x[j], _dot(i, u)
        sn = s - wp * (s - 2 * w[i] * rho * (1 - sq + 4.5 * cu * cu))
        dn = d - wm * (d - 6 * w[i] * rho * cu)
        if accel is not None:
            cf = _dot(i, f)
            sn = sn + (1 - 0.5 * wp) * 2 * w[i] * (9 * cu * cf - 3 * uf)
            dn = dn + (1 - 0.5 * wm) * 6 * w[i] * cf
        oi, oj = 0.5 * (sn + dn), 0.5 * (sn - dn)
        out[i] = oi if ns is None else (1 - ns) * oi + ns * x[j]
        out[j] = oj if ns is None else (1 - ns) * oj + ns * x[i]
    return out


def _stream(out, flags, lid):
    """Streaming with half-way bounce-back; `lid`: velocity of the walls with flag 2."""
    q = len(out)
    x = [out[0]] + [None] * (q - 1)
    for i in range(1, q):
        moved = _shift(out[i], _C[i])
        x[i] = moved if flags is None else torch.where(_shift(flags, _C[i]) != 0, out[_opp(i)], moved)
    return x if lid is None else _lid_links(x, flags, lid)


def _lid_links(x, flags, lid):
    """Momentum of the lid: links from walls with flag 2, which move at `lid` along x."""
    w, rho = _weights(len(x)), sum(x[1:], x[0])
    for i in range(1, len(x)):
        if _C[i][0]:
            link = _shift(flags, _C[i]) == 2
            x[i] = x[i] + torch.where(link, 6 * w[i] * rho * float(_C[i][0]) * lid, 0.0)
    return x


def _blocks(c, x, tau, accel, ns):
    """The collision over runs of planes, so that temporaries stay small beside the lattice."""
    nz, plane = c["nz"], c["nx"] * c["ny"]
    span = max(1, (1 << 23) // plane)
    for z in range(0, nz, span):
        part = slice(z, min(nz, z + span))
        a = None if accel is None else [v if not torch.is_tensor(v) or v.dim() == 0 else v[part] for v in accel]
        out = _collide(c, [v[part] for v in x], tau, a, None if ns is None else ns[part])
        for v, o in zip(x, out):
            v[part] = o
    return x


def _advance(c, x, tau, accel, flags, lid, steps):
    for _ in range(steps):
        x = _stream(_blocks(c, x, tau, accel, None), flags, lid)
        x = [v.contiguous() for v in x]
    return x


def _read(c, x, accel, flags):
    rho, u = _moments(x, len(x))
    if accel is not None:
        u = [v + 0.5 * a for v, a in zip(u, accel)]
    if flags is not None:
        fluid = (flags == 0).double()
        rho, u = rho * fluid, [v * fluid for v in u]
    return rho.reshape(-1), torch.stack([v.reshape(-1) for v in u])


def _voxels(c, tris, base):
    """`base` with 1 where a +x ray from the cell centre crosses the surface an odd number of times."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    t = torch.as_tensor(np.asarray(tris, np.float64).reshape(-1, 3, 3), device=DEVICE)
    a, b, d = t[:, 0], t[:, 1], t[:, 2]
    inside = torch.zeros((nz, ny, nx), dtype=torch.bool, device=DEVICE)
    yc = (torch.arange(ny, device=DEVICE, dtype=torch.float64) + 0.5) / ny + 1e-10 / nx
    area = (b[:, 1] - a[:, 1]) * (d[:, 2] - a[:, 2]) - (d[:, 1] - a[:, 1]) * (b[:, 2] - a[:, 2])
    for z in range(nz):
        p, yy = (z + 0.5) / nz + 2e-10 / nx, yc[:, None]
        v = ((yy - a[:, 1]) * (d[:, 2] - a[:, 2]) - (d[:, 1] - a[:, 1]) * (p - a[:, 2])) / area
        w = ((b[:, 1] - a[:, 1]) * (p - a[:, 2]) - (yy - a[:, 1]) * (b[:, 2] - a[:, 2])) / area
        row, tri = torch.nonzero((v >= 0) & (w >= 0) & (v + w <= 1), as_tuple=True)
        if row.numel() == 0:
            continue
        vv, ww = v[row, tri], w[row, tri]
        xh = a[tri, 0] + vv * (b[tri, 0] - a[tri, 0]) + ww * (d[tri, 0] - a[tri, 0])
        last = torch.ceil(xh * nx - 0.5).long().clamp(0, nx)  # cells left of the crossing flip
        count = torch.zeros((ny, nx + 1), dtype=torch.long, device=DEVICE)
        count.index_put_((row, last), torch.ones_like(last), accumulate=True)
        after = count.flip(1).cumsum(1).flip(1)  # crossings at or right of each cell
        inside[z] = (after[:, 1:] % 2) == 1
    return torch.where(inside, torch.ones_like(base), base)


def _sample(fields, at):
    """Trilinear values of the fields at points, with the corner indices and weights."""
    nz, ny, nx = fields[0].shape
    base = [torch.floor(p).long() for p in at]
    t = [p - b for p, b in zip(at, base)]
    corners, val = [], [0.0, 0.0, 0.0]
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                wt = 1.0
                for k, d in enumerate((dx, dy, dz)):
                    wt = wt * (t[k] if d else 1 - t[k])
                n = (((base[2] + dz) % nz) * ny + (base[1] + dy) % ny) * nx + (base[0] + dx) % nx
                corners.append((n, wt))
                val = [v + wt * f.reshape(-1)[n] for v, f in zip(val, fields)]
    return val, corners


def _coupled(c, seed, x, tau):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    cell = lambda v, a, s: torch.roll(v, -s, 2 - a)  # noqa: E731  value at the neighbour n + s e_a
    temp = torch.as_tensor(_temperature(c, seed), device=DEVICE).double().reshape(nz, ny, nx)
    g = [0.25 * temp] + [0.125 * temp] * 6
    i0 = _f32(nx / 2 + 0.25)
    left = torch.arange(nx, device=DEVICE, dtype=torch.float64)
    fill = (i0 - left).clamp(0, 1).expand(nz, ny, nx).contiguous()
    rec = torch.as_tensor(_particles(c, seed), device=DEVICE).float().double().T
    pos, vel, mass, resp = list(rec[:3]), list(rec[3:6]), rec[6], rec[7]
    force = [torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEVICE) for _ in range(3)]
    omega, dt, sigma = 1.0 / (0.5 + 4.0 * _f32(0.02)), 0.5, _f32(1e-4)
    for _ in range(c["steps"]):
        rho, u = _moments(x, len(x))
        u = [v + 0.5 * f for v, f in zip(u, force)]
        force = [torch.zeros_like(rho) for _ in range(3)]
        g = [_shift(g[i], _C[i]) for i in range(7)]
        temp = sum(g[1:], g[0])
        for i in range(7):
            cu = 0.0 if i == 0 else _dot(i, u)
            eq = (0.25 if i == 0 else 0.125) * temp * (1 + 4 * cu)
            g[i] = g[i] - omega * (g[i] - eq)
        force[1] = force[1] + _f32(1e-4) * (temp - 300.0)
        div = 0.0
        for a in range(3):
            face = 0.5 * (u[a] + cell(u[a], a, 1))
            flux = torch.where(face >= 0, face * fill, face * cell(fill, a, 1))
            div = div + flux - cell(flux, a, -1)
        fill = (fill - dt * div).clamp(0, 1)
        grad = [0.5 * (cell(fill, a, 1) - cell(fill, a, -1)) for a in range(3)]
        size = torch.sqrt(grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2)
        unit = [torch.where(size > 1e-12, v / size.clamp(min=1e-300), 0.0) for v in grad]
        curve = -0.5 * sum(cell(unit[a], a, 1) - cell(unit[a], a, -1) for a in range(3))
        force = [f + sigma * curve * v for f, v in zip(force, grad)]
        at = [torch.remainder(p, e) for p, e in zip(pos, (nx, ny, nz))]
        fu, corners = _sample(u, at)
        drag = [mass * (f - v) / resp for f, v in zip(fu, vel)]
        for n, wt in corners:
            for k in range(3):
                force[k].view(-1).index_put_((n,), -drag[k] * wt, accumulate=True)
        vel = [v + dt * d / mass for v, d in zip(vel, drag)]
        pos = [torch.remainder(p + dt * v, e) for p, v, e in zip(at, vel, (nx, ny, nz))]
        x = _advance(c, x, tau, force, None, None, 1)
    rho, u = _moments(x, len(x))
    u = [v + 0.5 * f for v, f in zip(u, force)]
    d = [[0.5 * (cell(u[b], a, 1) - cell(u[b], a, -1)) for a in range(3)] for b in range(3)]
    qc = 0.0
    for a in range(3):
        for b in range(3):
            qc = qc + 0.5 * ((0.5 * (d[a][b] - d[b][a])) ** 2 - (0.5 * (d[a][b] + d[b][a])) ** 2)
    points = torch.stack([*pos, *vel, mass, resp])
    return {"fill": fill.reshape(-1), "points": points, "q": qc.reshape(-1), "t": sum(g[1:], g[0]).reshape(-1),
            "rho": rho.reshape(-1), "u": torch.stack([v.reshape(-1) for v in u]), "f": None}


def _adjoint(c, seed, x, accel, flags):
    from torch.utils.checkpoint import checkpoint

    ns = _gray(c, seed).double().requires_grad_()
    tau = torch.tensor(_f32(c["tau"]), dtype=torch.float64, device=DEVICE, requires_grad=True)
    shape = (c["nz"], c["ny"], c["nx"])

    def step(n, t, *x):
        return tuple(_stream(_collide(c, list(x), t, accel, n.reshape(shape)), flags, None))

    for _ in range(c["steps"]):
        x = checkpoint(step, ns, tau, *x, use_reentrant=False)
    rho, u = _read(c, x, accel, flags)
    goal = _fields(c, seed)[1:].reshape(3, -1).double()
    grad_ns, grad_tau = torch.autograd.grad((u * goal).sum(), (ns, tau))
    return {"rho": rho.detach(), "u": u.detach(), "grad_ns": grad_ns, "grad_tau": grad_tau}


def exact(case, seed):
    c = case
    q = 19 if c["lattice"] == "d3q19" else 27
    cells = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "adjoint" and cells * q * 8 * (c["steps"] + 12) > 110e9:
        return None
    flags = _flags(c, seed)
    lid = _lid(seed) if c["geometry"] == "cavity" else None
    if c["kind"] == "body":
        flags = _voxels(c, _body(c, seed), _flags(dict(c, geometry="channel"), seed))
    fields = _fields(c, seed)
    x = [v.contiguous() for v in _equilibrium(fields[0].double(), [v.double() for v in fields[1:]], q)]
    del fields
    tau, accel = _f32(c["tau"]), None
    if c["force"]:
        accel = [_f32(c["force"]), 0.0, 0.0]
    if c["kind"] == "adjoint":
        return _adjoint(c, seed, x, accel, flags)
    if c["kind"] == "coupled":
        return _coupled(c, seed, x, tau)
    if lid is not None:
        x = _lid_links(x, flags, lid)  # the first step meets the moving wall too
    x = _advance(c, x, tau, accel, flags, lid, c["steps"])
    rho, u = _read(c, x, accel, flags)
    out = {"rho": rho, "u": u, "f": None}
    if c["kind"] == "monitored":
        speed2 = (u * u).sum(0)
        out["sums"] = [float(rho.sum()), float(0.5 * (rho * speed2).sum()), float(speed2.max().sqrt())]
    return out
