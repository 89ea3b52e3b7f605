"""The work that users of this package have it do, as cases that can be timed and checked.

Every case goes through a public entry point (the C ABI by way of ``capi.SW2Model``, or ``learned``):

* ``step``      one implicit time step (``load_state`` + ``step``, the state resident as in a time loop, or
                ``fe_newton`` on host arrays, the drop-in form), in the options of the time loop's default, of the
                FP64 benchmark path and of its FP32 path;
* ``residual``  the assembled residual: ``residual`` on host arrays, or the device-buffer form;
* ``jacobian``  the assembled CSR Jacobian on host arrays;
* ``bicgstab``  the reference's preconditioned BiCGStab on a caller's system;
* ``guess``     inference of the learned initial guess from two resident states;
* ``gradient``  one training pass of its network: forward, loss and backward.

A mesh is generated once per size and its model (sparsity, maps, hierarchy) built once, as a run does; the seed
makes the states on it.  ``exact`` evaluates the same quantities in 64 bits with torch alone.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os

import numpy as np
import torch

GRAVITY = 9.8
HERE = os.path.dirname(os.path.abspath(__file__))
WEIGHTS = os.path.join(os.path.dirname(HERE), "adh_kraken_b200", "weights", "basin_guess.npz")

# The benchmark's options for its FP64 and FP32 paths (GMRES(100) + AMG, relative Newton test); the time loop's
# default is the reference's absolute test with GMRES(30) + AMG.
_BENCH = dict(tol_nonlin=1e-8, tol_nonlin_rel=1e-8, inc_nonlin=1e-6, max_nonlin_it=10, krylov_max_it=20000,
              krylov_tol=1e-6, precond=2, krylov_method=1, krylov_restart=100)
OPTIONS = {
    "default": {},
    "plain": dict(_BENCH, krylov_precision=64),
    "fast": dict(_BENCH, krylov_precision=32, krylov_basis_precision=32),
    "mixed": dict(_BENCH, krylov_precision=32, krylov_basis_precision=64),
    # the reference's Krylov method, converged tightly: what a run compared with the reference asks for
    "parity": dict(krylov_method=0, krylov_tol=1e-12, tol_nonlin=1e-11, inc_nonlin=1e-9, max_nonlin_it=15),
}


def listed():
    return [
        # the CPU-runnable flume: every array in L1/L2, a step is launches and latency
        {"name": "flume_step_default", "kind": "step", "mesh": "flume", "nx": 101, "ny": 11, "opts": "default", "api": "host"},
        # a small wet/dry beach with both boundary kinds, at the size and settings of the parity tests
        {"name": "wetdry_step_parity", "kind": "step", "mesh": "wetdry", "nx": 24, "ny": 24, "opts": "parity", "api": "host"},
        # the tidal basin, coarse: a calibration run's grid, FP64 throughout
        {"name": "basin125k_step_plain", "kind": "step", "mesh": "basin", "nx": 251, "ny": 251, "opts": "plain", "api": "host"},
        # the tidal basin at the configured million triangles, FP32 cycles in FP64 refinement: the production path
        {"name": "basin1M_step_fast", "kind": "step", "mesh": "basin", "nx": 707, "ny": 707, "opts": "fast", "api": "resident"},
        # the same path at the benchmark's four million triangles
        {"name": "basin4M_step_fast", "kind": "step", "mesh": "basin", "nx": 1414, "ny": 1414, "opts": "fast", "api": "resident"},
        # assemble_residual as the reference's Newton calls it on the flume (host arrays, latency)
        {"name": "flume_residual_host", "kind": "residual", "mesh": "flume", "nx": 101, "ny": 11, "api": "host"},
        # the residual on device buffers, wet/dry beach, close to that entry point's limit
        {"name": "beach126k_residual_device", "kind": "residual", "mesh": "beach", "nx": 505, "ny": 126, "api": "device"},
        # assemble_jacobian as the reference's Newton calls it, wet/dry beach
        {"name": "beach250k_jacobian_host", "kind": "jacobian", "mesh": "beach", "nx": 709, "ny": 177},
        # the reference's linear solver entry on the flume's system at a 10 s step, block ILU(0)
        {"name": "flume_bicgstab_ilu", "kind": "bicgstab", "mesh": "flume", "nx": 101, "ny": 11, "precond": 1},
        # inference of the guess on the basin it was trained for
        {"name": "basin1M_guess", "kind": "guess", "mesh": "basin", "nx": 707, "ny": 707},
        # the training experiment's small basin: one pass is launches
        {"name": "basin3k_gradient", "kind": "gradient", "mesh": "basin", "nx": 40, "ny": 40},
        # training on a half-resolution basin
        {"name": "basin250k_gradient", "kind": "gradient", "mesh": "basin", "nx": 354, "ny": 354},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "residual", "jacobian", "bicgstab", "guess", "gradient"])
    case = {"kind": kind}
    if kind == "step":
        opts = rng.choice(["default", "parity", "plain", "fast", "fast", "mixed"])
        mesh = {"default": rng.choice(["flume", "basin"]), "parity": "wetdry"}.get(opts, "basin")
        if mesh == "flume":
            nx, ny = _log_int(rng, 41, 401), _log_int(rng, 5, 21)
        elif mesh == "wetdry":
            nx = ny = _log_int(rng, 12, 24)
        else:
            nx = ny = _log_int(rng, 32, {"default": 120, "plain": 707, "fast": 1200, "mixed": 707}[opts])
        case.update(mesh=mesh, nx=nx, ny=ny, opts=opts, api=rng.choice(["host", "resident"]))
    elif kind == "residual":
        api = rng.choice(["host", "device"])
        ny = _log_int(rng, 8, 126 if api == "device" else 250)
        case.update(mesh=rng.choice(["beach", "basin"]), nx=4 * ny + rng.randrange(2), ny=ny, api=api)
    elif kind == "jacobian":
        ny = _log_int(rng, 8, 180)
        case.update(mesh=rng.choice(["beach", "basin"]), nx=4 * ny + rng.randrange(2), ny=ny)
    elif kind == "bicgstab":
        case.update(mesh="flume", nx=_log_int(rng, 21, 121), ny=_log_int(rng, 5, 11), precond=rng.choice([0, 1, 2]))
    else:
        nx = ny = _log_int(rng, 24, 1000 if kind == "guess" else 354)
        case.update(mesh="basin", nx=nx, ny=ny)
    return case


# ------------------------------------------------------------------------------------------------ meshes and states

def _size(case):
    nx, ny = case["nx"], case["ny"]
    return nx * ny, 2 * (nx - 1) * (ny - 1)


def _domain(mesh, nx, ny):
    """Lengths and time step of a mesh kind."""
    if mesh == "flume":
        return 10.0 * (nx - 1), 10.0 * (ny - 1), 60.0
    if mesh == "wetdry":
        return 1000.0 * (nx - 1) / 23.0, 1000.0 * (ny - 1) / 23.0, 30.0
    if mesh == "basin":
        return 20000.0, 20000.0, 300.0
    return 40000.0, 10000.0, 120.0                     # beach


@functools.lru_cache(maxsize=2)
def _mesh(mesh, nx, ny):
    """Nodes (x-major), triangles and boundary strings: a rectangle's grid with its interior nodes moved by up to a
    fifth of a spacing and each quad cut along a random diagonal (node degrees 4 to 8, as in an unstructured mesh)."""
    rng = np.random.default_rng(1000 * nx + ny)
    lx, ly, _ = _domain(mesh, nx, ny)
    jitter = 0.0 if mesh == "flume" else 0.2
    i, j = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    inside = (i > 0) & (i < nx - 1) & (j > 0) & (j < ny - 1)
    x = (i + np.where(inside, rng.uniform(-jitter, jitter, i.shape), 0.0)).ravel() * (lx / (nx - 1))
    y = (j + np.where(inside, rng.uniform(-jitter, jitter, i.shape), 0.0)).ravel() * (ly / (ny - 1))
    a = (i[:-1, :-1] * ny + j[:-1, :-1]).ravel()
    b, c, d = a + ny, a + ny + 1, a + 1                # counter-clockwise round the quad
    flip = rng.random(a.size) < 0.5
    t0 = np.stack([a, b, np.where(flip, d, c)], axis=1)
    t1 = np.stack([np.where(flip, b, a), c, d], axis=1)
    tri = np.stack([t0, t1], axis=1).reshape(-1, 3).astype(np.int32)
    if mesh == "flume":
        z = -1e-4 * x
    elif mesh == "wetdry":
        z = -2.0 + 2.6 * x / lx + rng.normal(0.0, 0.05, x.shape)
    elif mesh == "basin":
        z = np.full_like(x, -10.0)
        for k in range(8):
            cx, cy = rng.uniform(0, lx), rng.uniform(0, ly)
            r2 = (x - cx) ** 2 + (y - cy) ** 2
            z += rng.uniform(1, 5) * np.exp(-r2 / (2 * rng.uniform(500, 2000) ** 2)) * np.clip(x / 3000.0, 0.0, 1.0) * 0.7
    else:
        z = -20.0 + 23.0 * x / lx + rng.normal(0.0, 0.2, x.shape)
    west = np.arange(ny)
    z[west] = {"flume": 0.0, "wetdry": -2.0, "basin": -10.0, "beach": -20.0}[mesh]
    out_west = np.stack([west[1:], west[:-1]], axis=1)
    seg, kind = [out_west], [np.full(ny - 1, 1 if mesh == "basin" else 0)]
    if mesh == "flume":                                # depth at the outlet
        east = (nx - 1) * ny + np.arange(ny)
        seg.append(np.stack([east[:-1], east[1:]], axis=1)); kind.append(np.ones(ny - 1))
    elif mesh == "wetdry":                             # depth along a third of the south edge
        south = np.arange(nx // 3 + 1) * ny
        seg.append(np.stack([south[:-1], south[1:]], axis=1)); kind.append(np.ones(nx // 3))
    elif mesh == "basin":                              # inflow on the east edge
        east = (nx - 1) * ny + np.arange(ny)
        seg.append(np.stack([east[:-1], east[1:]], axis=1)); kind.append(np.zeros(ny - 1))
    return (np.ascontiguousarray(np.stack([x, y, z], axis=1)), tri, np.concatenate(seg).astype(np.int32),
            np.concatenate(kind).astype(np.int32))


def _waves(rng, x, y, lx, ly, size, count=4):
    """A few long waves with random phases, quiet at the west edge."""
    f = np.zeros_like(x)
    for _ in range(count):
        kx, ky = rng.integers(1, 4), rng.integers(0, 4)
        f += rng.uniform(-1, 1) * np.sin(2 * np.pi * kx * x / lx + rng.uniform(0, 6.28)) * np.cos(np.pi * ky * y / ly)
    return size * f * np.clip(4.0 * x / lx, 0.0, 1.0) / math.sqrt(count)


def _inputs(case, seed):
    """Three time levels of the state and the boundary values of the coming step, from the seed."""
    mesh, nx, ny = case["mesh"], case["nx"], case["ny"]
    xyz = _mesh(mesh, nx, ny)[0]
    lx, ly, dt = _domain(mesh, nx, ny)
    rng = np.random.default_rng([seed, nx, ny])
    x, y, z = xyz[:, 0], xyz[:, 1], xyz[:, 2]
    n = x.size
    still = {"flume": 2.0 + 0 * z, "wetdry": 0.1 - z}.get(mesh, -z)
    # amplitudes of h, u, v; of their change over a step; of that change's change (the basin's: a solved tidal run's)
    amp = {"flume": ((0.02, 0.02, 0.02), (2e-3, 2e-3, 2e-3), (2e-4, 2e-4, 2e-4)),
           "wetdry": ((0.01, 0.02, 0.02), (1e-3, 2e-3, 2e-3), (1e-4, 2e-4, 2e-4)),
           "basin": ((0.15, 0.12, 0.006), (0.03, 6e-3, 3e-4), (2.4e-3, 2e-3, 6e-5)),
           "beach": ((0.1, 0.05, 0.05), (1e-2, 5e-3, 5e-3), (1e-3, 5e-4, 5e-4))}[mesh]
    base, drift, bend = ([_waves(rng, x, y, lx, ly, a) for a in part] for part in amp)
    levels = []
    for k in range(3):                                 # the newest first
        s = np.empty(3 * n)
        for v in range(3):
            s[v::3] = (still if v == 0 else 0.0) + base[v] - k * drift[v] + 0.5 * k * (k - 1) * bend[v]
        if mesh in ("wetdry", "beach"):                # velocities die out on the dry part
            wet = still > 0.05
            s[1::3] *= wet
            s[2::3] *= wet
        if case["kind"] in ("residual", "jacobian", "bicgstab"):   # a Newton iterate is rougher than a solved state
            s += 1e-3 * rng.standard_normal(3 * n)
        levels.append(s)
    bc = {"flume": (2.0 + 0.01 * rng.uniform(-1, 1), 0.25 + 0.02 * rng.uniform(-1, 1), 0.0),
          "wetdry": (2.1 + 0.02 * rng.uniform(-1, 1), 0.05 + 0.01 * rng.uniform(-1, 1), 0.01),
          "basin": (10.0 + 0.05 * rng.uniform(-1, 1), -0.01 * rng.uniform(0.1, 1), 0.0),
          "beach": (20.0, 0.003 + 0.005 * rng.uniform(), 0.0)}[mesh]
    return levels, dt, bc


def _case_object(case):
    from adh_kraken_b200.mesh import SW2Case
    xyz, tri, seg, kind = _mesh(case["mesh"], case["nx"], case["ny"])
    return SW2Case(case["mesh"], xyz, tri, seg, kind, np.zeros(3 * len(xyz)), 1.0, 1, {})


@functools.lru_cache(maxsize=2)
def _model(mesh, nx, ny):
    from adh_kraken_b200.capi import SW2Model
    return SW2Model(_case_object({"mesh": mesh, "nx": nx, "ny": ny}))


@functools.lru_cache(maxsize=2)
def _guesser(mesh, nx, ny):
    from adh_kraken_b200 import learned
    return learned.Guesser(learned.Net.load(WEIGHTS), _case_object({"mesh": mesh, "nx": nx, "ny": ny}))


class _Resident:
    """A device array of the library as torch sees it."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": "<f8", "version": 3}


def prepare(case, seed):
    key = case["mesh"], case["nx"], case["ny"]
    levels, dt, bc = _inputs(case, seed)
    state = {"case": case, "dt": dt, "bc": bc}
    if case["kind"] in ("guess", "gradient"):
        g = state["guesser"] = _guesser(*key)
        state["levels"] = [torch.from_numpy(s).cuda() for s in levels]
        if case["kind"] == "gradient":
            from adh_kraken_b200 import learned
            state["workspace"] = learned.Workspace(g.graph.n, train=True)
        return state
    state["model"] = _model(*key)
    if case["kind"] == "step":
        from adh_kraken_b200.capi import default_opts
        state["opts"] = default_opts(**OPTIONS[case["opts"]])
        if case["api"] == "resident":                  # page-locked, as a program that keeps its state on the GPU would
            levels = [torch.from_numpy(s).pin_memory().numpy() for s in levels]
    elif case["kind"] == "residual" and case["api"] == "device":
        levels = [torch.from_numpy(s).cuda() for s in levels]
        state["out"] = torch.empty(levels[0].numel(), dtype=torch.float64, device="cuda")
    elif case["kind"] == "bicgstab":
        state["system"] = [t.cpu().numpy() for t in _linear_system(case, seed)[:3]]
    state["levels"] = levels
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "guess":
        g, (now, before, _) = state["guesser"], state["levels"]
        g.predict_ptr(now.data_ptr(), before.data_ptr(), torch.cuda.current_stream().cuda_stream)
        return g.guess
    if kind == "gradient":
        return _gradient(state)
    m = state["model"]
    m.set_step(state["dt"], *state["bc"])
    if kind == "step":
        now, before, oldest = state["levels"]
        if case["api"] == "host":
            sol, st = m.fe_newton(now, before, np.zeros(m.ndofs, np.int32), opts=state["opts"])
            return {"sol": sol, "success": st["success"]}
        m.load_state(now, before, oldest)
        st = m.step(state["opts"])
        sol = torch.as_tensor(_Resident(m.device_state()[0], m.ndofs), device="cuda")
        return {"sol": sol, "success": st["success"]}
    if kind == "residual":
        if case["api"] == "host":
            return m.residual(*state["levels"])
        from adh_kraken_b200.capi import lib
        m._check(lib().sw2g_assemble_residual_noalloc(m.h, *(ctypes.c_void_p(t.data_ptr()) for t in state["levels"]),
                                                      ctypes.c_void_p(state["out"].data_ptr())))
        return state["out"]
    if kind == "jacobian":
        return m.jacobian(*state["levels"])
    vals, b, scale = state["system"]
    x, _, _ = m.bicgstab(vals, b, np.zeros(m.ndofs), scale, max_it=4000, tol=1e-12, precond=case["precond"])
    return x


def _gradient(state):
    """One training pass as learned.train makes it, up to the weight update."""
    from adh_kraken_b200 import learned as L
    g, ws, (after, now, before) = state["guesser"], state["workspace"], state["levels"]
    net, n, lib, p = g.net, g.graph.n, L._L(), L._p
    L._check(lib.sw2n_features(n, p(now), p(before), p(g.z), p(net.mu), p(net.sd), p(ws.F), None), "features")
    L._check(lib.sw2n_targets(n, p(after), p(now), p(before), p(net.scale), L.MIN_DEPTH, p(ws.T), p(ws.M), None), "targets")
    L.forward(net, g.graph, ws, train=True)
    parts = L._check(lib.sw2n_mse(n, p(ws.Y), p(ws.T), p(ws.M), p(ws.dY), p(ws.lpart), None), "loss")
    L.backward(net, g.graph, ws)
    return {"correction": ws.Y, "gradient": net.g, "loss": ws.lpart[:parts].sum()}


def work(case):
    """Bytes: each input read once and each output written once (a step: also its two Jacobians, built and read once
    each).  Operations: the element formulas (~700 a residual, 18 residuals a Jacobian), and a dense layer's products."""
    V, T = _size(case)
    nnz = 9 * (7 * V)
    mesh, state = 92 * T, 24 * V
    kind = case["kind"]
    if kind == "residual":
        return {"bytes": mesh + 4 * state, "flops": 700 * T}
    if kind == "jacobian":
        return {"bytes": mesh + 3 * state + 8 * nnz, "flops": 18 * 700 * T}
    if kind == "step":
        return {"bytes": mesh + 4 * state + 2 * (2 * 8 * nnz), "flops": 2 * 18 * 700 * T + 4 * nnz}
    if kind == "bicgstab":
        return {"bytes": 12 * nnz + 3 * state, "flops": 4 * nnz}
    dense = 2 * V * (8 * 64 + 3 * 256 * 64 + 64 * 3)
    graph = 4 * 7 * V * 4
    if kind == "guess":
        return {"bytes": 3 * state + graph, "flops": dense}
    return {"bytes": 3 * state + graph + 4 * 50000, "flops": 3 * dense}


# ------------------------------------------------------------------------------------------- the same in 64 bits

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Elements:
    """Triangles of a mesh with P1 geometry, and the SW2 element residual (SUPG, wet/dry by cutting along h = 0)."""

    def __init__(self, case, device=None):
        xyz, tri, seg, kind = _mesh(case["mesh"], case["nx"], case["ny"])
        d = device or _dev()
        self.n, self.tri = len(xyz), torch.from_numpy(tri).long().to(d)
        self.seg, self.kind = torch.from_numpy(seg).long().to(d), torch.from_numpy(kind).to(d)
        p = torch.from_numpy(xyz).to(d)
        self.x, self.z = p[self.tri][:, :, :2], p[self.tri][:, :, 2]
        self.area, self.g = _geometry(self.x)
        a, b = p[self.seg[:, 0], :2], p[self.seg[:, 1], :2]
        self.len = (b - a).norm(dim=1)
        self.nrm = torch.stack([b[:, 1] - a[:, 1], a[:, 0] - b[:, 0]], dim=1) / self.len[:, None]
        # integrals of products of three P1 functions over a triangle of unit area: 6, 2 or 1 sixtieths
        t = torch.tensor([[[6 if i == j == k else 1 if len({i, j, k}) == 3 else 2 for k in range(3)] for j in range(3)]
                          for i in range(3)], dtype=torch.float64)
        self.triple = (t / 60.0).to(d)

    def flags(self, now, old):
        """Triangles that are dry at both levels: their old levels add no mass."""
        h, ho = now.view(-1, 3)[:, 0][self.tri], old.view(-1, 3)[:, 0][self.tri]
        return ((h < 0) & (ho < 0)).all(dim=1)

    def residual(self, h, v, ho, vo, hoo, voo, dry, dt, pressure=True):
        """[T,3,3] (vertex; h, u, v) of the states' depths [T,3] and velocities [T,3,2]."""
        g, x, A, grav = self.g, self.x, self.area, GRAVITY
        r = torch.zeros(len(A), 3, 3, dtype=torch.float64, device=A.device)
        wet, old, older = _Cut(x, h, A), _Cut(x, ho, A), _Cut(x, hoo, A)

        def convection(ar, gr, hh, vv):
            q = torch.einsum("abc,ta,tbi,tcj->tij", self.triple, hh, vv, vv) * ar[:, None, None]
            m = (hh.sum(1, keepdim=True) + hh)[:, :, None] * vv
            mass = torch.einsum("tak,tk->ta", gr, m.sum(1) * ar[:, None] / 12.0)
            return torch.cat([mass[:, :, None], torch.einsum("tak,tik->tai", gr, q)], dim=2) * -dt

        def storage(ar, gr, hh, vv):
            out = torch.zeros_like(r)
            out[:, :, 0] = ar[:, None] / 12.0 * (hh.sum(1, keepdim=True) + hh)
            return out

        def average(ar, gr, hh, vv):
            return ar[:, None] * torch.cat([hh.mean(1, keepdim=True), vv.mean(1)], dim=1)

        r = r + wet.vertexwise(convection, g, h, v)
        lump = A[:, None, None] / 3.0
        for cut, hh, vv, w, mass in ((wet, h, v, 1.0, True), (old, ho, vo, -1.0, ~dry), (older, hoo, voo, 0.0, ~dry)):
            s = w * cut.vertexwise(storage, g, hh, vv)
            r = r + (s if mass is True else s * mass[:, None, None])
            r[:, :, 1:] += lump * w * cut.fraction[:, None, None] * vv * hh.clamp(min=1e-6)[:, :, None]
        resist = 0.002 / (2.0 * grav)
        f = v * v.norm(dim=2, keepdim=True)
        r[:, :, 1:] += (dt * grav * resist * wet.fraction * A / 12.0)[:, None, None] * (f.sum(1, keepdim=True) + f)
        grad_z, grad_h = torch.einsum("ta,tak->tk", self.z, g), torch.einsum("ta,tak->tk", h, g)
        if pressure:
            def forces(ar, gr, hh, vv, xx):
                out = torch.zeros_like(r)
                sq = ((hh * hh).sum(1) + hh[:, 0] * hh[:, 1] + hh[:, 1] * hh[:, 2] + hh[:, 0] * hh[:, 2]) * ar / 6.0
                out[:, :, 1:] = -0.5 * grav * dt * gr * sq[:, None, None]
                out[:, :, 1:] += grav * dt * (ar[:, None] / 12.0 * (hh.sum(1, keepdim=True) + hh))[:, :, None] * grad_z[:, None, :]
                for a, b in ((0, 1), (1, 2), (2, 0)):
                    nrm = torch.stack([xx[:, b, 1] - xx[:, a, 1], xx[:, a, 0] - xx[:, b, 0]], dim=1)
                    qa = 3 * hh[:, a] ** 2 + 2 * hh[:, a] * hh[:, b] + hh[:, b] ** 2
                    qb = hh[:, a] ** 2 + 2 * hh[:, a] * hh[:, b] + 3 * hh[:, b] ** 2
                    out[:, a, 1:] += 0.5 * grav * dt / 12.0 * qa[:, None] * nrm
                    out[:, b, 1:] += 0.5 * grav * dt / 12.0 * qb[:, None] * nrm
                return out
            r = r + wet.vertexwise(forces, g, h, v, places=True)
        # SUPG
        mean_new, mean_old = wet.total(average, g, h, v), old.total(average, g, ho, vo)
        frac = torch.where(wet.fraction > 0, wet.fraction, torch.ones_like(A))
        on = wet.fraction > 0
        mean = torch.where(on[:, None], mean_new / (A * frac)[:, None], torch.zeros_like(mean_new))
        hm, um = mean[:, 0], mean[:, 1:]
        hden = hm.clamp(min=1.1920928955078125e-07)
        tau = 0.5 * (A * old.fraction.clamp(min=0)).sqrt() / ((um * um).sum(1) + grav * hden + 2.220446049250313e-16).sqrt()

        def transport(ar, gr, hh, vv):
            ha, ua = hh.mean(1), vv.mean(1)
            dh, dv = torch.einsum("ta,tak->tk", hh, gr), torch.einsum("tai,tak->tik", vv, gr)
            c = (ua * dh).sum(1) + ha * (dv[:, 0, 0] + dv[:, 1, 1])
            return (ar * dt)[:, None] * torch.cat([c[:, None], torch.einsum("tk,tik->ti", ua, dv)], dim=1)

        eq = mean_new - mean_old + wet.total(transport, g, h, v, nodal=True)
        fac = wet.fraction[:, None]
        speed = um.norm(dim=1, keepdim=True)
        eq[:, 1:] += A[:, None] * dt * fac * grav * (grad_h + grad_z + resist * um * speed / hden[:, None])
        c, m = eq[:, 0], eq[:, 1:]
        t = torch.where(hm.abs() >= 2.220446049250313e-16, tau, torch.zeros_like(tau))
        flux = um * c[:, None] + hm[:, None] * m
        r[:, :, 0] += t[:, None] * torch.einsum("tak,tk->ta", g, flux)
        own = (grav * hm * c)[:, None] + um * hm[:, None] * m
        r[:, :, 1] += t[:, None] * (g[:, :, 0] * own[:, None, 0] + g[:, :, 1] * (um[:, 1] * hm * m[:, 0])[:, None])
        r[:, :, 2] += t[:, None] * (g[:, :, 1] * own[:, None, 1] + g[:, :, 0] * (um[:, 0] * hm * m[:, 1])[:, None])
        return r

    def boundary(self, h, v, dt, bc, pressure=True):
        """[S,2,3] of the strings: a velocity string (0) or a depth string (1)."""
        depth, vx, vy = bc
        given = torch.tensor([vx, vy], dtype=torch.float64, device=h.device)
        is_vel = (self.kind == 0)[:, None]
        hh = torch.where(is_vel, h, torch.full_like(h, depth))
        vv = torch.where(is_vel[:, :, None], given.expand_as(v), v)
        nrm, ln = self.nrm, self.len
        vn = torch.einsum("tak,tk->ta", vv, nrm)
        out = torch.zeros(len(ln), 2, 3, dtype=torch.float64, device=h.device)
        m2 = torch.tensor([[[3.0, 1.0], [1.0, 1.0]], [[1.0, 1.0], [1.0, 3.0]]], dtype=torch.float64, device=h.device) / 12.0
        m3 = torch.tensor([[[[12., 3, ], [3, 2]], [[3, 2], [2, 3]]], [[[3., 2], [2, 3]], [[2, 3], [3, 12]]]],
                          dtype=torch.float64, device=h.device) / 60.0
        out[:, :, 0] = torch.einsum("abc,tb,tc->ta", m2, hh, vn) * ln[:, None]
        carried = vv * (vn >= 2.220446049250313e-16)[:, :, None]
        out[:, :, 1:] = torch.einsum("abcd,tbi,tc,td->tai", m3, carried, vn, hh) * ln[:, None, None]
        if pressure:
            sq = torch.einsum("abc,tb,tc->ta", m2, hh, hh) - torch.einsum("abc,tb,tc->ta", m2, h, h)
            out[:, :, 1:] += torch.where(is_vel, torch.zeros_like(sq), 0.5 * GRAVITY * sq * ln[:, None])[:, :, None] * nrm[:, None, :]
        shut = (~is_vel[:, 0]) & ((h < 2.220446049250313e-16).any(dim=1) | (depth < 2.220446049250313e-16))
        return dt * out * (~shut)[:, None, None]

    def assemble(self, now, old, older, dry, dt, bc):
        s, o, p = (t.view(-1, 3) for t in (now, old, older))
        e = [q for t in (s, o, p) for q in (t[:, 0][self.tri], t[:, 1:][self.tri])]
        out = torch.zeros(self.n, 3, dtype=torch.float64, device=now.device)
        out.index_add_(0, self.tri.reshape(-1), -self.residual(*e, dry, dt).reshape(-1, 3))
        b = self.boundary(s[:, 0][self.seg], s[:, 1:][self.seg], dt, bc)
        out.index_add_(0, self.seg.reshape(-1), -b.reshape(-1, 3))
        return out.reshape(-1)

    def jacobian(self, now, old, older, dry, dt, bc):
        """CSR values of the central differences, and the node pattern (rows, columns, position of each node pair)."""
        s, o, p = (t.view(-1, 3) for t in (now, old, older))
        n, dev = self.n, now.device
        keys = torch.cat([(self.tri[:, :, None] * n + self.tri[:, None, :]).reshape(-1),
                          (self.seg[:, :, None] * n + self.seg[:, None, :]).reshape(-1)])
        pairs, at = torch.unique(keys, return_inverse=True)
        blocks = torch.zeros(len(pairs), 3, 3, dtype=torch.float64, device=dev)
        done = 0
        for ids, f, first in ((self.tri, self.residual, True), (self.seg, self.boundary, False)):
            k = ids.shape[1]
            h, v = s[:, 0][ids], s[:, 1:][ids]
            rest = (o[:, 0][ids], o[:, 1:][ids], p[:, 0][ids], p[:, 1:][ids], dry, dt) if first else (dt, bc)
            place = at[done:done + ids.numel() * k].view(-1, k, k)
            done += ids.numel() * k
            for b in range(k):
                for w in range(3):
                    u = h[:, b] if w == 0 else v[:, b, w - 1]
                    eps = (u.abs() * (1.0 + 1e-4) - u.abs()).clamp(min=1e-4)
                    side = []
                    for sign in (1.0, -1.0):
                        h2, v2 = h.clone(), v.clone()
                        if w == 0:
                            h2[:, b] += sign * eps
                        else:
                            v2[:, b, w - 1] += sign * eps
                        side.append(f(h2, v2, *rest, pressure=w == 0))
                    col = (side[0] - side[1]) / (2.0 * eps)[:, None, None]
                    for a in range(k):
                        blocks[:, :, w].index_add_(0, place[:, a, b], col[:, a])
        rows, cols = pairs // n, pairs % n
        deg = torch.bincount(rows, minlength=n)
        start = torch.cat([torch.zeros(1, dtype=torch.long, device=dev), (9 * deg).cumsum(0)])
        slot = torch.arange(len(pairs), device=dev) - torch.cat([torch.zeros(1, dtype=torch.long, device=dev), deg.cumsum(0)])[rows]
        pos = (start[rows] + 3 * slot)[:, None, None] + (3 * deg[rows])[:, None, None] * torch.arange(3, device=dev)[None, :, None] \
            + torch.arange(3, device=dev)[None, None, :]
        vals = torch.zeros(9 * len(pairs), dtype=torch.float64, device=dev)
        vals[pos.reshape(-1)] = blocks.reshape(-1)
        return vals, rows, cols, pos


def _geometry(x):
    a, b = x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]
    area = 0.5 * (a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0])
    nxt, prv = x[:, [1, 2, 0]], x[:, [2, 0, 1]]
    e = nxt - prv
    safe = torch.where(area == 0, torch.ones_like(area), area)
    return area, torch.stack([e[:, :, 1], -e[:, :, 0]], dim=2) * 0.5 / safe[:, None, None]


class _Cut:
    """The wet part of triangles: the whole, minus the dry corner, the wet corner, or nothing."""

    def __init__(self, x, h, area):
        self.x, self.area = x, area
        dry = h <= 0
        self.count = dry.sum(1)
        odd = torch.where((self.count == 1)[:, None], dry, ~dry).to(torch.float64)
        self.corner = odd.argmax(1)
        pick = torch.nn.functional.one_hot(self.corner, 3).bool()
        ho = (h * pick).sum(1, keepdim=True)
        cut = ((self.count == 1) | (self.count == 2))[:, None] & ~pick
        self.pick, self.xi = pick, torch.where(cut, h / torch.where(cut, h - ho, torch.ones_like(h)), torch.zeros_like(h))
        self.sub_x = self.interp(x)
        self.sub_h = torch.where(pick, h, torch.zeros_like(h))
        self.sub_area, self.sub_g = _geometry(self.sub_x)
        part = self.sub_area / area
        one, two = self.count == 1, self.count == 2
        thin = part < 2.220446049250313e-16
        self.use = ((one | two) & ~thin).to(torch.float64)
        self.full = (self.count <= 1).to(torch.float64)
        self.sign = torch.where(two, 1.0, -1.0).to(torch.float64) * self.use
        self.fraction = torch.where(self.count == 0, 1.0, 0.0).to(torch.float64)
        self.fraction = torch.where(one, torch.where(thin, 1.0, 1.0 - part), self.fraction)
        self.fraction = torch.where(two, torch.where(thin, 0.0, part), self.fraction)

    def interp(self, f):
        xi = self.xi if f.dim() == 2 else self.xi[:, :, None]
        at = f.gather(1, self.corner[:, None] if f.dim() == 2 else self.corner[:, None, None].expand(-1, 1, f.shape[2]))
        return f + xi * (at - f)

    def _both(self, fn, g, h, v, nodal, places):
        sub = (self.sub_area, self.sub_g, self.interp(h) if nodal else self.sub_h, self.interp(v))
        if places:
            return fn(self.area, g, h, v, self.x), fn(*sub, self.sub_x)
        return fn(self.area, g, h, v), fn(*sub)

    def total(self, fn, g, h, v, nodal=False):
        """An element quantity [T,k] over the wet part."""
        whole, sub = self._both(fn, g, h, v, nodal, False)
        return self.full[:, None] * whole + torch.where(self.use[:, None] > 0, self.sign[:, None] * sub, torch.zeros_like(sub))

    def vertexwise(self, fn, g, h, v, places=False):
        """Vertex contributions [T,3,3]; a cut vertex hands its share beyond the cut back to the corner."""
        whole, sub = self._both(fn, g, h, v, False, places)
        xo = self.x.gather(1, self.corner[:, None, None].expand(-1, 1, 2))
        far = (self.x - xo).norm(dim=2)
        xi = torch.where(self.pick, torch.ones_like(far), (self.sub_x - xo).norm(dim=2) / torch.where(far == 0, torch.ones_like(far), far))
        back = ((1.0 - xi)[:, :, None] * sub).sum(1, keepdim=True)
        moved = xi[:, :, None] * sub + self.pick[:, :, None] * back
        return self.full[:, None, None] * whole + torch.where(self.use[:, None, None] > 0, self.sign[:, None, None] * moved, torch.zeros_like(moved))


def _linear_system(case, seed):
    """(CSR values, right-hand side, scale factors, dense matrix) of a Newton correction, symmetrically scaled."""
    levels, _, bc = _inputs(case, seed)
    dt = 10.0
    el = _Elements(case, "cpu")                        # its sums run in one order there
    s, o, p = (torch.from_numpy(t).to(el.area.device) for t in levels)
    dry = el.flags(s, o)
    b = el.assemble(s, o, p, dry, dt, bc)
    vals, rows, cols, pos = el.jacobian(s, o, p, dry, dt, bc)
    three = torch.arange(3, device=s.device)
    i = (3 * rows)[:, None, None] + three[None, :, None] + 0 * pos
    j = (3 * cols)[:, None, None] + three[None, None, :] + 0 * pos
    biggest = torch.zeros_like(b).scatter_reduce_(0, i.reshape(-1), vals[pos].abs().reshape(-1), "amax")
    scale = 1.0 / biggest.sqrt()
    vals[pos] = vals[pos] * scale[i] * scale[j]
    dense = torch.zeros(len(b), len(b), dtype=torch.float64, device=s.device)
    dense[i, j] = vals[pos]
    return vals, b * scale, scale, dense


def _newton(case, seed):
    """The step's solution: Newton with the difference Jacobian and dense solves until it no longer improves."""
    levels, dt, bc = _inputs(case, seed)
    el = _Elements(case)
    old, older = (torch.from_numpy(t).to(el.area.device) for t in levels[:2])
    sol = old.clone()
    fixed = torch.zeros(el.n, 3, dtype=torch.bool, device=sol.device)
    fixed[:, 1:] |= (old.view(-1, 3)[:, :1] <= 0)
    fixed = fixed.view(-1)
    sol[fixed] = 0.0
    dry = el.flags(old, old)
    three, best, kept = torch.arange(3, device=sol.device), math.inf, sol
    for _ in range(30):
        r = el.assemble(sol, old, older, dry, dt, bc)
        vals, rows, cols, pos = el.jacobian(sol, old, older, dry, dt, bc)
        dense = torch.zeros(len(sol), len(sol), dtype=torch.float64, device=sol.device)
        dense[(3 * rows)[:, None, None] + three[None, :, None] + 0 * pos, (3 * cols)[:, None, None] + three[None, None, :] + 0 * pos] = vals[pos]
        fixed |= dense.diagonal().abs() < 2.220446049250313e-16
        free = (~fixed).nonzero()[:, 0]
        size = float(r[free].abs().max())
        if size < best:
            best, kept = size, sol.clone()
        elif best < 1e-10:
            break
        sol = sol.clone()
        sol[free] += torch.linalg.solve(dense[free][:, free], r[free])
    return kept


def _network(case, seed, train):
    """The message-passing network in 64 bits: the guess, or (correction, gradient, loss)."""
    levels, _, _ = _inputs(case, seed)
    xyz, tri, _, _ = _mesh(case["mesh"], case["nx"], case["ny"])
    d, f8 = _dev(), torch.float64
    w = np.load(WEIGHTS)
    mu, sd, scale = (torch.from_numpy(w[k]).to(d, f8) for k in ("mu", "sd", "scale"))
    flat, at, layers = torch.from_numpy(w["w"]).to(d), 0, []
    for i, o in ((8, 64), (256, 64), (256, 64), (256, 64), (64, 3)):
        layers.append((flat[at:at + i * o].bfloat16().to(f8).view(o, i).requires_grad_(train),
                       flat[at + i * o:at + i * o + o].to(f8).requires_grad_(train)))
        at += i * o + o
    states = [torch.from_numpy(s).to(d).view(-1, 3) for s in levels]
    after, now, before = states if train else (None, states[0], states[1])
    n = len(now)
    e = np.concatenate([tri[:, [0, 1]], tri[:, [1, 2]], tri[:, [2, 0]]]).astype(np.int64)
    key = torch.unique(torch.from_numpy(np.concatenate([e[:, 0] * n + e[:, 1], e[:, 1] * n + e[:, 0]])).to(d))
    src, dst = key // n, key % n
    deg = torch.bincount(src, minlength=n).to(f8)
    xy = torch.from_numpy(xyz[:, :2].copy()).to(d)
    step = xy[dst] - xy[src]
    step = (step / (step.norm(dim=1).mean() * deg[src][:, None])).float().to(f8)     # the graph's weights are FP32
    inv = (1.0 / deg).float().to(f8)

    def gather(values, out):
        return torch.zeros(n, out, dtype=f8, device=d).index_add(0, src, values)

    f = torch.cat([now, now - before, torch.from_numpy(xyz[:, 2:].copy()).to(d), (now[:, :1] > 0).to(f8)], dim=1)
    silu = torch.nn.functional.silu
    x = silu(((f - mu) / sd) @ layers[0][0].T + layers[0][1])
    for W, b in layers[1:4]:
        diff = x[dst] - x[src]
        feats = torch.cat([x, gather(x[dst], 64) * inv[:, None], gather(step[:, :1] * diff, 64), gather(step[:, 1:] * diff, 64)], dim=1)
        x = x + silu(feats @ W.T + b)
    y = x @ layers[4][0].T + layers[4][1]
    for _ in range(2):
        y = (y + gather(y[dst], 3)) / (deg + 1.0)[:, None]
    if not train:
        guess = 2.0 * now - before + scale * y
        keep = ~(now[:, 0] > 0.05) | ~(guess[:, 0] > 0.05)
        return torch.where(keep[:, None], now, guess).reshape(-1)
    mask = ((now[:, 0] > 0.05) & (after[:, 0] > 0.05)).to(f8)
    err = (y - (after - 2.0 * now + before) / scale) * mask[:, None]
    loss = (err * err).sum() / (3 * n)
    loss.backward()
    grad = torch.cat([torch.cat([W.grad.reshape(-1), b.grad]) for W, b in layers])
    return {"correction": y.detach(), "gradient": grad, "loss": loss.detach()}


def exact(case, seed):
    kind = case["kind"]
    V, T = _size(case)
    if kind == "guess":
        with torch.no_grad():
            return _network(case, seed, False)
    if kind == "gradient":
        return _network(case, seed, True)
    if kind == "step":                                 # by dense factorisation, while that is quick
        return {"sol": _newton(case, seed), "success": None} if V <= 1500 else None
    if kind == "bicgstab":
        vals, b, scale, dense = _linear_system(case, seed)
        return torch.linalg.solve(dense, b) * scale
    levels, dt, bc = _inputs(case, seed)
    el = _Elements(case)
    s, o, p = (torch.from_numpy(t).to(el.area.device) for t in levels)
    dry = el.flags(s, o)
    return el.assemble(s, o, p, dry, dt, bc) if kind == "residual" else el.jacobian(s, o, p, dry, dt, bc)[0]
