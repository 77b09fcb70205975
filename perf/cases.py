"""The work that users of this framework have it do, as measurable cases.

A case names one call of the public interface and its sizes: whole timesteps of
a scene (``Simulation.run``, ``Ensemble.run``), the plug-in methods that a host
code binds one by one (diffusion, turbulence model, pressure solve) and the
learned initial guess (network inference and one training step).  ``listed()``
gives the fixed ones, ``draw()`` others of the same ranges.  ``exact()`` restates
the plug-in methods and the network in 64-bit torch, without this package.
"""
import ctypes as C
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

import artss_b200 as A
from artss_b200 import learned, scenes
from artss_b200.ensemble import Ensemble

H = 0.0375  # cell size of the plume scenes (m)
FT_U, FT_P = 1, 4
NU, KAPPA, CS, DT = 3.1e-5, 4.2e-5, 0.2, 0.005
STATE = ("u", "v", "w", "p", "T", "nu_t")
KEPT = ("u", "v", "w", "u0", "v0", "w0", "u_tmp", "v_tmp", "w_tmp", "p", "p0", "T", "T0", "T_tmp", "f_x", "f_y", "f_z")
AGAIN = 64  # steps after which a scene goes back to the state it was prepared in, so that every pass is the same work


def listed():
    return [
        # a small room with a door, seven touching walls, Jacobi diffusion: launches and latency count
        {"name": "step_room32", "kind": "step", "scene": "room", "nx": 32, "ny": 32, "nz": 32, "levels": 2,
         "diffusion": "Jacobi", "graphs": False},
        # the closed plume box, stepped one by one, as the command line does
        {"name": "step_plume64", "kind": "step", "scene": "plume", "nx": 64, "ny": 64, "nz": 64, "levels": 4,
         "diffusion": "ColoredGaussSeidel", "graphs": False},
        # the channel with a cube that bench.py times, whole-step graphs: a production run
        {"name": "step_channel256", "kind": "step", "scene": "channel", "nx": 256, "ny": 128, "nz": 128, "levels": 4,
         "diffusion": "ColoredGaussSeidel", "graphs": True},
        # a parameter study: plume boxes of several sizes side by side, mixed-precision pressure
        {"name": "ensemble8", "kind": "ensemble", "count": 8, "largest": 96, "first": 0},
        # velocity diffusion of one component, turbulent, sides that are no multiple of a tile
        {"name": "diffuse_cgs_turb", "kind": "diffuse", "method": "cgs", "turb": True, "nx": 200, "ny": 104, "nz": 72},
        # the same on odd sides and laminar
        {"name": "diffuse_cgs_odd", "kind": "diffuse", "method": "cgs", "turb": False, "nx": 161, "ny": 97, "nz": 49},
        # Jacobi diffusion, the solver of most of the shipped configurations
        {"name": "diffuse_jacobi_turb", "kind": "diffuse", "method": "jacobi", "turb": True, "nx": 128, "ny": 128,
         "nz": 128},
        # one later-step pressure call of the FP64 V-cycle solver on the benchmark's grid
        {"name": "pressure_vcycle", "kind": "pressure", "nx": 256, "ny": 128, "nz": 128, "levels": 4},
        # the mixed-precision Poisson solve to 1e-8, pure Neumann with box obstacles
        {"name": "poisson_mixed256", "kind": "poisson", "n": 256, "levels": 5, "obstacles": True},
        # the dynamic Smagorinsky model
        {"name": "dynamic_smagorinsky", "kind": "dynamic", "nx": 192, "ny": 96, "nz": 96},
        # the learned guess: inference on the plume channel's grid
        {"name": "unet_forward", "kind": "unet", "D": 64, "H": 64, "W": 128, "train": False},
        # one training step: forward, loss, backward, Adam
        {"name": "unet_train", "kind": "unet", "D": 32, "H": 32, "W": 64, "train": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "diffuse", "diffuse", "pressure", "poisson", "dynamic", "unet", "ensemble"])
    if kind == "step":
        scene = rng.choice(["room", "plume", "channel"])
        if scene == "room":
            n = rng.choice([32, 64])
            return {"kind": kind, "scene": scene, "nx": n, "ny": n, "nz": n, "levels": 2,
                    "diffusion": rng.choice(["Jacobi", "ColoredGaussSeidel"]), "graphs": rng.random() < 0.5}
        if scene == "channel":
            n = rng.choice([64, 128, 256])
            return {"kind": kind, "scene": scene, "nx": n, "ny": n // 2, "nz": n // 2, "levels": rng.choice([3, 4]),
                    "diffusion": "ColoredGaussSeidel", "graphs": rng.random() < 0.5}
        s = [16 * _log(rng, 1, 10) for _ in range(3)]
        return {"kind": kind, "scene": scene, "nx": s[0], "ny": s[1], "nz": s[2], "levels": rng.choice([3, 4]),
                "diffusion": rng.choice(["ColoredGaussSeidel", "ColoredGaussSeidel", "Jacobi"]),
                "graphs": rng.random() < 0.5}
    if kind == "diffuse":
        s = [_log(rng, 17, 200) for _ in range(3)]
        return {"kind": kind, "method": rng.choice(["cgs", "jacobi"]), "turb": rng.random() < 0.6, "nx": s[0],
                "ny": s[1], "nz": s[2]}
    if kind == "pressure":
        s = [16 * _log(rng, 2, 10) for _ in range(3)]
        return {"kind": kind, "nx": s[0], "ny": s[1], "nz": s[2], "levels": rng.choice([3, 4])}
    if kind == "poisson":
        return {"kind": kind, "n": 32 * rng.randint(2, 7), "levels": 5, "obstacles": rng.random() < 0.5}
    if kind == "dynamic":
        s = [_log(rng, 17, 112) for _ in range(3)]
        return {"kind": kind, "nx": s[0], "ny": s[1], "nz": s[2]}
    if kind == "unet":
        return {"kind": kind, "D": 4 * rng.randint(4, 14), "H": 32 * rng.randint(1, 2), "W": rng.choice([64, 128]),
                "train": rng.random() < 0.4}
    return {"kind": kind, "count": rng.randint(2, 6), "largest": rng.choice([48, 64, 96]), "first": rng.randint(0, 99)}


# ------------------------------------------------------------------ inputs


class _View:
    """Device memory of the library as a torch tensor, which keeps its owner."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _tensor(ptr, shape, owner):
    return torch.as_tensor(_View(int(ptr), tuple(shape), owner), device="cuda")


def _addr(p):
    return C.cast(p, C.c_void_p).value


def _waves(seed, dims, count, longest=3):
    """`count` smooth fields of unit RMS plus 5% noise on a grid of dims = (nz, ny, nx) inner cells and one ghost layer."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    ax = [(torch.arange(n + 2, device="cuda", dtype=torch.float64) - 0.5) / n for n in dims]
    out = []
    for _ in range(count):
        f = torch.zeros([n + 2 for n in dims], device="cuda", dtype=torch.float64)
        for _ in range(6):
            k = torch.randint(1, longest + 1, (3,), generator=g, device="cuda").double() * math.pi
            ph = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) * 2 * math.pi
            s = [torch.sin(k[a] * ax[a] + ph[a]) for a in range(3)]
            f += s[0][:, None, None] * s[1][None, :, None] * s[2][None, None, :]
        f += 0.05 * torch.randn(f.shape, generator=g, device="cuda", dtype=torch.float64)
        out.append(f / f.square().mean().sqrt())
    return out


def _ghosts(x, sign, value=0.0):
    """Ghost planes of a closed box, patch after patch: x[ghost] = sign x[neighbour] + 2 value."""
    for a in (2, 1, 0):
        n = x.shape[a]
        x.select(a, 0).copy_(sign * x.select(a, 1) + 2 * value)
        x.select(a, n - 1).copy_(sign * x.select(a, n - 2) + 2 * value)
    return x


def _box(nx, ny, nz, levels):
    ext = (nx * H, ny * H, nz * H)
    return scenes.Scene(nx=nx, ny=ny, nz=nz, X=(0.0, ext[0]), Y=(0.0, ext[1]), Z=(0.0, ext[2]), dt=DT, steps=10 ** 7,
                        n_level=levels, boundaries=scenes.closed_box_bcs())


def _write(sc):
    fd, path = tempfile.mkstemp(suffix=".xml")
    os.close(fd)
    return scenes.write(sc, path)


def _scene(case, seed):
    rng = random.Random(seed)
    kw = dict(steps=10 ** 7, n_level=case["levels"], diffusion=case["diffusion"], seed=seed)
    if case["scene"] == "room":
        return scenes.room_with_door(n=case["nx"], hrr=rng.uniform(25.0, 75.0), **kw)
    if case["scene"] == "channel":
        return scenes.channel_with_cube(nx=case["nx"], ny=case["ny"], nz=case["nz"], hrr=rng.uniform(50.0, 150.0), **kw)
    sc = _box(case["nx"], case["ny"], case["nz"], case["levels"])
    sc.diffusion, sc.seed, sc.hrr = case["diffusion"], seed, rng.uniform(10.0, 50.0)
    sc.source_pos = (0.5 * sc.X[1], 0.5 * sc.Y[1], 0.15 * sc.Z[1])
    return sc


def _start(sim, sc, seed):
    """A flow under way: smooth velocities of about 0.3 m/s, then the steps whose pressure solve starts from nothing."""
    dims = [sc.nz, sc.ny, sc.nx]
    for name, f in zip("uvw", _waves(seed, dims, 3)):
        f = (0.3 * f).reshape(-1).cpu().numpy()
        for field in (name, name + "0", name + "_tmp"):
            sim.set_field(field, f)
    sim.run(4)


class _Run:
    """A simulation under way, its fields on the device, and a copy of its state."""

    def __init__(self, sim, sc, seed):
        _start(sim, sc, seed)
        self.sim, self.steps = sim, 0
        self.out = {f: _tensor(sim.device_pointer(f), (sim.size,), sim) for f in STATE}
        self.kept = [(sim.device_pointer(f), _tensor(sim.device_pointer(f), (sim.size,), sim).clone()) for f in KEPT]

    def back(self):
        """The prepared state again, every AGAIN steps."""
        if self.steps == AGAIN:
            lib, at = A.load_cuda(), C.POINTER(C.c_double)
            for p, t in self.kept:
                A.cuda_check(lib.artss_copy(self.sim.context, C.cast(p, at), C.cast(t.data_ptr(), at), 0), "copy")
            self.steps = 0
        self.steps += 1


class _Scene:
    """A context of one scene with its level lists, and device arrays; freed with the object."""

    def __init__(self, sc):
        self.sc, path = sc, _write(sc)
        self.geom = A.Geometry(path)
        os.unlink(path)
        self.ctx = A.Context(self.geom)
        self.lib, self.h = self.ctx.lib, self.ctx.h
        self.shape = (self.ctx.grid.Nz[0], self.ctx.grid.Ny[0], self.ctx.grid.Nx[0])
        self.solver, self.free = C.c_void_p(), None

    def field(self, values=None):
        return self.ctx.field(None if values is None else values.reshape(-1).cpu().numpy())

    def view(self, p):
        return _tensor(_addr(p), self.shape, self)

    def __del__(self):
        if sys.is_finalizing():
            return
        if self.solver and self.free:
            self.free(self.solver)
        self.geom.close()
        self.ctx.close()


def _diffuse_inputs(case, seed):
    """(u, nu_t, viscosity): a velocity component with its wall values, a turbulent viscosity"""
    dims = [case["nz"], case["ny"], case["nx"]]
    x, e = _waves(seed, dims, 2)
    return _ghosts(0.3 * x, -1.0), _ghosts(1e-3 * e.square(), 1.0)


def _dynamic_inputs(case, seed):
    return [_ghosts(0.3 * f, -1.0) for f in _waves(seed, [case["nz"], case["ny"], case["nx"]], 3)]


def _pressure_inputs(case, seed):
    """a pressure of an earlier step and a divergence"""
    p, d = _waves(seed, [case["nz"], case["ny"], case["nx"]], 2)
    rhs = torch.zeros_like(d)
    i = (slice(1, -1),) * 3
    rhs[i] = d[i] - d[i].mean()
    return _ghosts(0.05 * p, 1.0), rhs


def _poisson_solution(case, seed):
    """the solution that the right-hand side is made of: smooth modes and grid-scale noise"""
    n = case["n"]
    p = _waves(seed, [n] * 3, 1)[0] * (n / 16.0)
    p += 0.2 * _waves(seed + 1, [n] * 3, 1, longest=n // 4)[0]
    return _ghosts(p, 1.0)


def _unet_inputs(case, seed):
    """network input (residual, fluid mask, right-hand side in channels 0..2) and target"""
    dims = [case["D"], case["H"], case["W"]]
    r, b, t = (f[1:-1, 1:-1, 1:-1].float() for f in _waves(seed, dims, 3))
    x = torch.zeros(dims + [16], device="cuda", dtype=torch.bfloat16)
    x[..., 0], x[..., 1], x[..., 2] = r.bfloat16(), 1.0, b.bfloat16()
    return x, 0.1 * t


def _biases(seed):
    """biases as a network under training has them"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [0.2 * torch.randn(cout, generator=g, device="cuda") for _, cout, _, _ in LAYERS]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        sc = _scene(case, seed)
        path = _write(sc)
        sim = A.Simulation(path)
        os.unlink(path)
        sim.set_graphs(case["graphs"])
        return {"kind": kind, "run": _Run(sim, sc, seed)}
    if kind == "ensemble":
        sizes = [s for s in (32, 48, 64, 96) if s <= case["largest"]]
        members = scenes.plume_ensemble(count=case["count"], seed=case["first"], steps=10 ** 7, sizes=sizes)
        paths = []
        for n, sc in enumerate(members):
            rng = random.Random(1000 * seed + n)
            sc.seed, sc.hrr = rng.randint(0, 10 ** 6), rng.uniform(10.0, 150.0)
            paths.append(_write(sc))
        ens = Ensemble(paths, graphs=True)
        for path in paths:
            os.unlink(path)
        return {"kind": kind, "ens": ens, "runs": [_Run(s, m, seed + n) for n, (s, m) in enumerate(zip(ens.sims, members))]}
    if kind == "unet":
        st = _Scene(scenes.plume_box(n=16, steps=1, n_level=2))
        net = learned.UNet(st.ctx, (case["D"], case["H"], case["W"]), seed=seed)
        for layer, b in zip(net.layers, _biases(seed)):
            layer.b.copy_(b)
        x, t = _unet_inputs(case, seed)
        return {"kind": kind, "train": case["train"], "scene": st, "net": net, "x": x.reshape(-1), "t": t.reshape(-1).contiguous()}
    if kind == "poisson":
        sc = scenes.poisson_boxes(n=case["n"], seed=2, n_level=case["levels"])
        if not case["obstacles"]:
            sc.obstacles = []
        st = _Scene(sc)
        p, b = st.field(_poisson_solution(case, seed)), st.field()
        A.cuda_check(st.lib.artss_laplacian(st.h, b, p, 0), "laplacian")
        cfg = A.MixedCfg(case["levels"], 2, 1, A.MIXED_REMOVE_MEAN, 6.0 / 7.0, 0.0, 1e-2, 20, 1e-8, 200)
        A.cuda_check(st.lib.artss_mixed_create(st.h, C.byref(cfg), C.byref(st.solver)), "mixed")
        st.free = st.lib.artss_mixed_destroy
        return {"kind": kind, "scene": st, "p": p, "b": b, "stats": A.SolveStats(), "out": st.view(p)}
    st = _Scene(_box(case["nx"], case["ny"], case["nz"], case.get("levels", 0)))
    if kind == "diffuse":
        x, e = _diffuse_inputs(case, seed)
        return {"kind": kind, "scene": st, "cgs": case["method"] == "cgs", "x": st.field(x),
                "ev": st.field(e) if case["turb"] else None, "u": (u := st.field()), "u0": st.field(),
                "cfg": A.IterCfg(100, 1e-7, 1.0), "stats": A.IterStats(), "out": st.view(u)}
    if kind == "dynamic":
        ev = st.field()
        return {"kind": kind, "scene": st, "uvw": [st.field(f) for f in _dynamic_inputs(case, seed)], "ev": ev,
                "out": st.view(ev)}
    p0, rhs = _pressure_inputs(case, seed)
    cfg = A.MgCfg(case["levels"], 2, 100, 2, 1e-8, 0, 0, 100, 1e-8, 0.6666666667)
    A.cuda_check(st.lib.artss_mg_create(st.h, C.byref(cfg), C.byref(st.solver)), "mg")
    st.free = st.lib.artss_mg_destroy
    p = st.field()
    return {"kind": kind, "scene": st, "p0": st.field(p0), "rhs": st.field(rhs), "p": p, "stats": A.MgStats(),
            "out": st.view(p)}


def run(state):
    kind = state["kind"]
    if kind == "step":
        r = state["run"]
        r.back()
        r.sim.run(1)
        return r.out
    if kind == "ensemble":
        for r in state["runs"]:
            r.back()
        state["ens"].run(1)
        return [r.out for r in state["runs"]]
    if kind == "unet":
        net = state["net"]
        out = net.forward(state["x"])
        if not state["train"]:
            return out
        loss = net.loss_grad(state["t"], state["t"].numel())
        net.backward()
        net.adam(lr=1e-3)
        return {"out": out, "loss": loss, "grads": [g for layer in net.layers for g in layer.grads],
                "weights": [p for layer in net.layers for p in layer.params]}
    st = state["scene"]
    lib, h = st.lib, st.h
    if kind == "diffuse":
        if state["cgs"]:
            # as the solver calls it: out and in coupled from one field, in scratch afterwards
            A.cuda_check(lib.artss_couple(h, state["x"], state["u0"], state["u"], *[None] * 6), "couple")
            A.cuda_check(lib.artss_diffuse_cgs(h, state["u"], state["u0"], state["x"], NU, state["ev"], DT, FT_U,
                                               C.byref(state["cfg"]), 3, C.byref(state["stats"])), "diffuse")
        else:
            A.cuda_check(lib.artss_couple(h, state["x"], state["u0"], state["u"], *[None] * 6), "couple")
            A.cuda_check(lib.artss_diffuse_jacobi(h, state["u"], state["u0"], state["x"], NU, state["ev"], DT, FT_U,
                                                  C.byref(state["cfg"]), C.byref(state["stats"])), "diffuse")
    elif kind == "dynamic":
        A.cuda_check(lib.artss_turb_dynamic_smagorinsky(h, state["ev"], *state["uvw"], NU), "dynamic smagorinsky")
    elif kind == "pressure":
        A.cuda_check(lib.artss_copy(h, state["p"], state["p0"], 0), "copy")
        A.cuda_check(lib.artss_mg_pressure(st.solver, state["p"], state["rhs"], 0, C.byref(state["stats"])), "pressure")
    else:
        A.cuda_check(lib.artss_fill(h, state["p"], 0, 0.0), "fill")
        A.cuda_check(lib.artss_mixed_solve(st.solver, state["p"], state["b"], C.byref(state["stats"])), "mixed solve")
    return state["out"]


# ------------------------------------------------------------------ work and tolerance


def _members(case):
    sizes = [s for s in (32, 48, 64, 96) if s <= case["largest"]]
    return scenes.plume_ensemble(count=case["count"], seed=case["first"], sizes=sizes)


def work(case):
    kind = case["kind"]
    if kind in ("step", "ensemble"):
        n = case["nx"] * case["ny"] * case["nz"] if kind == "step" else sum(s.inner_cells() for s in _members(case))
        # the state (u, v, w, p, T) in, it and nu_t out; about 1000 operations a cell and step
        return {"bytes": 88.0 * n, "flops": 1000.0 * n}
    if kind == "unet":
        # multiply-adds of the ten convolutions per level-0 voxel, three times as many with both gradients
        v = case["D"] * case["H"] * case["W"]
        macs = 27 * (16 * 16 * 3 + 48 * 16 + (16 * 32 + 32 * 32 * 2 + 96 * 32) / 8 + (32 * 64 + 64 * 64) / 64)
        params = 27 * (16 * 16 * 3 + 48 * 16 + 16 * 32 + 32 * 32 * 2 + 96 * 32 + 32 * 64 + 64 * 64)
        t = case["train"]
        return {"bytes": v * 64.0 + params * (4.0 if not t else 28.0), "flops": 2.0 * macs * v * (3 if t else 1)}
    if kind == "poisson":
        n = case["n"] ** 3
        return {"bytes": 16.0 * n, "flops": 2000.0 * n}  # some 15 cycles
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "diffuse":
        return {"bytes": (24.0 if case["turb"] else 16.0) * n, "flops": (30.0 if case["turb"] else 16.0) * 4 * n}
    if kind == "dynamic":
        return {"bytes": 32.0 * n, "flops": 1400.0 * n}  # 20 filters and the average, 27 cells each
    return {"bytes": 24.0 * n, "flops": 150.0 * n}  # two V-cycles


def tolerance(case):
    return TOLERANCE[case["kind"]]


TOLERANCE = {
    # FP64 sums in another order, a step or a solve long
    "step": {"rel": 1e-12, "max": 1e-10},
    "diffuse": {"rel": 2e-15, "max": 2e-14},
    "pressure": {"rel": 5e-14, "max": 5e-13},
    # the coefficient is a quotient that is large where its denominator is small
    "dynamic": {"rel": 1e-12, "max": 1e-9},
    # solved to a relative residual of 1e-8, which bounds the solution less tightly
    "poisson": {"rel": 1e-6, "max": 3e-6},
    "ensemble": {"rel": 1e-6, "max": 1e-4},
    # BF16 activations through ten layers
    "unet": {"rel": 2e-2, "max": 0.5},
}


# ------------------------------------------------------------------ 64 bits


def _sides(x):
    """inner values and the six face neighbours' (x-, x+, y-, y+, z-, z+)"""
    i = slice(1, -1)
    return x[i, i, i], (x[i, i, :-2], x[i, i, 2:], x[i, :-2, i], x[i, 2:, i], x[:-2, i, i], x[2:, i, i])


def _exact_diffuse(case, seed):
    b, e = _diffuse_inputs(case, seed)
    i = (slice(1, -1),) * 3
    a = (NU + e[i] if case["turb"] else torch.full_like(b[i], NU)) * DT / (H * H)
    rb = 1.0 + 6.0 * a
    x = b.clone()
    k = sum(torch.meshgrid(*[torch.arange(1, n - 1, device=x.device) for n in x.shape], indexing="ij"))
    masks = [(k % 2 == 0), (k % 2 == 1)] if case["method"] == "cgs" else [torch.ones_like(k, dtype=torch.bool)]
    for _ in range(100):
        old = x[i].clone()
        for m in masks:
            _, n = _sides(x)
            new = (b[i] + a * ((n[1] + n[0]) + (n[3] + n[2]) + (n[5] + n[4]))) / rb
            x[i] = torch.where(m, new, x[i])
        res = (rb * (x[i] - old)).square().sum().sqrt()
        _ghosts(x, -1.0)
        if float(res) <= 1e-7:
            break
    return x


def _filter(f):
    w = (0.25, 0.5, 0.25)
    out = torch.zeros_like(f)
    n = f.shape
    out[1:-1, 1:-1, 1:-1] = sum(w[a] * w[b] * w[c] * f[c:n[0] - 2 + c, b:n[1] - 2 + b, a:n[2] - 2 + a]
                                for a in range(3) for b in range(3) for c in range(3))
    return out


def _exact_dynamic(case, seed):
    i = (slice(1, -1),) * 3
    f = [_filter(x) for x in _dynamic_inputs(case, seed)]

    def d(x, axis):  # axis 0: x
        _, n = _sides(x)
        return (n[2 * axis + 1] - n[2 * axis]) * 0.5 / H

    def pad(x):
        out = torch.zeros_like(f[0])
        out[i] = x
        return out

    pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    s = [pad(0.5 * (d(f[a], b) + d(f[b], a))) for a, b in pairs]
    weight = (1, 1, 1, 2, 2, 2)
    norm = lambda t: (2.0 * sum(w * x * x for w, x in zip(weight, t))).sqrt()  # noqa: E731
    sb = norm(s)
    fs = [_filter(x) for x in s]
    sbf = norm(fs)
    delta = (H * H * H) ** (1.0 / 3.0)
    low, m = [], []
    for n, (a, b) in enumerate(pairs):
        uv = pad((f[a] * f[b])[i])
        low.append((0.0 if n == 4 else _filter(uv)) - uv)  # the filter of u w is never formed
        m.append(2.0 * delta * delta * (_filter(pad((sb * s[n])[i])) - 4.0 * sbf * fs[n]))

    def combine(p):
        return p[0] + p[1] * p[2] + 2.0 * p[3] + 2.0 * p[4] + 2.0 * p[5]

    cs = combine([x * y for x, y in zip(low, m)]) / combine([y * y for y in m])
    cs = pad(cs[i])
    # the average of 27 cells runs in place in list order: cell after cell along i + 2 j + 4 k
    nz, ny, nx = (n - 2 for n in cs.shape)
    flat = cs.reshape(-1)
    grid = torch.meshgrid(*[torch.arange(1, n + 1, device=cs.device) for n in (nz, ny, nx)], indexing="ij")
    at = (grid[2] + (nx + 2) * (grid[1] + (ny + 2) * grid[0])).reshape(-1)
    t = (grid[2] + 2 * grid[1] + 4 * grid[0]).reshape(-1)
    order = torch.argsort(t)
    at, count = at[order], torch.bincount(t).tolist()
    off = torch.tensor([a + (nx + 2) * (b + (ny + 2) * c) for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)],
                       device=cs.device)
    begin = 0
    for n in count:
        q = at[begin:begin + n]
        flat[q] = flat[q[:, None] + off[None, :]].sum(1) / 27.0
        begin += n
    ev = 2.0 * cs * delta * delta * sb
    return pad(torch.where(ev + NU < 0, torch.zeros_like(ev), ev)[i])


def _exact_pressure(case, seed):
    p, rhs = _pressure_inputs(case, seed)
    L, w = case["levels"], 0.6666666667
    i = (slice(1, -1),) * 3

    def stencil(x, level):
        c, n = _sides(x)
        return sum(n) / (H * 2.0 ** level) ** 2, c

    def jacobi(x, b, level):
        s, c = stencil(x, level)
        out = x.clone()
        out[i] = (1 - w) * c + w * (s - b[i]) * (H * 2.0 ** level) ** 2 / 6.0
        return _ghosts(out, 1.0)

    def residual(x, b, level):
        s, c = stencil(x, level)
        return b[i] - (s - 6.0 * c / (H * 2.0 ** level) ** 2)

    def smooth(x, b, level):  # two relaxations, of which the second is not kept
        return jacobi(_ghosts(x, 1.0), b, level)

    def solve(x, b, level):
        x, it, res, last = _ghosts(x, 1.0), 0, 1e4, x
        while res > 1e-8 and it < 100:
            last, x = x, jacobi(x, b, level)
            res = float(residual(x, b, level).square().sum().sqrt())
            it += 1
        return x if it % 2 else last

    def pad(x):
        out = torch.zeros([n + 2 for n in x.shape], dtype=x.dtype, device=x.device)
        out[i] = x
        return out

    def prolong(e):
        shape = [2 * (n - 2) for n in e.shape]
        out = torch.zeros(shape, dtype=e.dtype, device=e.device)

        def at(x, axis, s):  # the neighbour on side s along axis, or the cell itself (s = 0)
            return x.narrow(axis, 1 + s, x.shape[axis] - 2)

        for a in (0, 1):
            for b in (0, 1):
                for c in (0, 1):
                    v = e
                    for axis, side in ((0, c), (1, b), (2, a)):
                        v = 0.75 * at(v, axis, 0) + 0.25 * at(v, axis, 1 if side else -1)
                    out[c::2, b::2, a::2] = v
        return pad(out)

    for _ in range(2):
        e, r = [p], [rhs]
        for level in range(L):
            e[level] = smooth(e[level], r[level], level)
            q = residual(e[level], r[level], level)
            q = q.reshape(q.shape[0] // 2, 2, q.shape[1] // 2, 2, q.shape[2] // 2, 2).mean((1, 3, 5))
            r.append(pad(q))
            e.append(torch.zeros_like(r[-1]))
        for level in range(L, 0, -1):
            up = e[level - 1] + _ghosts(prolong(e[level]), 1.0)
            e[level - 1] = solve(up, r[level - 1], level - 1) if level == L else smooth(up, r[level - 1], level - 1)
        p = _ghosts(e[0], 1.0)
    return p


LAYERS = [(16, 16, True, 3), (16, 16, True, 16), (16, 32, True, 16), (32, 32, True, 32), (32, 64, True, 32),
          (64, 64, True, 64), (96, 32, True, 96), (32, 32, True, 32), (48, 16, True, 48), (16, 16, False, 16)]


def _exact_unet(case, seed):
    rng = np.random.default_rng(seed)
    weights = []
    for (cin, cout, _, real), b in zip(LAYERS, _biases(seed)):
        w = np.zeros((27, cout, cin), np.float32)
        w[:, :, :real] = rng.standard_normal((27, cout, real)) * np.sqrt(2.0 / (27 * real))
        weights.append([torch.from_numpy(w).double().cuda().requires_grad_(case["train"]),
                        b.double().requires_grad_(case["train"])])
    x, target = _unet_inputs(case, seed)
    x = x.double()

    def conv(n, v):
        (w, b), d = weights[n], v.shape
        q = torch.nn.functional.pad(v, (0, 0, 1, 1, 1, 1, 1, 1))
        y = b
        for t in range(27):
            y = y + q[t // 9:t // 9 + d[0], t // 3 % 3:t // 3 % 3 + d[1], t % 3:t % 3 + d[2]] @ w[t].T
        return torch.relu(y) if LAYERS[n][2] else y

    def pool(v):
        d = v.shape
        return v.reshape(d[0] // 2, 2, d[1] // 2, 2, d[2] // 2, 2, d[3]).mean((1, 3, 5))

    def up(v):
        return v.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)

    s0 = conv(1, conv(0, x))
    s1 = conv(3, conv(2, pool(s0)))
    b2 = conv(5, conv(4, pool(s1)))
    d1 = conv(7, conv(6, torch.cat([up(b2), s1], -1)))
    out = conv(9, conv(8, torch.cat([up(d1), s0], -1)))
    if not case["train"]:
        return out.reshape(-1)
    loss = 0.5 * (out[..., 0] - target.double()).square().mean()
    flat = [p for layer in weights for p in layer]
    grads = torch.autograd.grad(loss, flat)
    # Adam's first step: both moments, corrected, are the gradient and its square
    new = [p.detach() - 1e-3 * g / (g.abs() + 1e-8) for p, g in zip(flat, grads)]
    return {"out": out.detach().reshape(-1), "loss": float(loss), "grads": list(grads), "weights": new}


def exact(case, seed):
    """64-bit results of the plug-in methods and the network.  None for whole timesteps (a plain restatement takes
    minutes) and for pressure problems with obstacles."""
    kind = case["kind"]
    if kind == "diffuse":
        return _exact_diffuse(case, seed)
    if kind == "dynamic":
        return _exact_dynamic(case, seed)
    if kind == "pressure":
        return _exact_pressure(case, seed)
    if kind == "poisson" and not case["obstacles"]:
        p = _poisson_solution(case, seed)
        return _ghosts(p - p[1:-1, 1:-1, 1:-1].mean(), 1.0)
    if kind == "unet":
        return _exact_unet(case, seed)
    return None
