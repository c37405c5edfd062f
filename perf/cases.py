"""The measured workloads: whole steps of the multi-layer XPBD solver through
its public entry points, over the sizes that the scene generators, the tests
and the benchmark of this repository use.

A pass is what a user's frame loop does: some time steps, then the state (the
host-buffer path returns it with every step).  An FP32 solver holds its state
in FP32 and the ABI widens it to double, so the state of those cases is
returned as the FP32 values it is.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from multilayersolver2024_b200 import (MLX_ENERGY_NEOHOOKEAN, MLX_ENERGY_STVK_VOIGT, MLX_FP32, MLX_FP64, ContactSet,
                                       Mesh3D, Solver, StepCache, XpbdLayer3D, find_boundary_vertices, scenes,
                                       to_lame)
from multilayersolver2024_b200.contacts import PlaneContactFinder3D, SphereContactFinder, find_contacts
from multilayersolver2024_b200.learned import Mlp
from multilayersolver2024_b200.warm_start_training import load_warm_start
from multilayersolver2024_b200.xpbd_layer3d import ResidentSim


def listed():
    return [
        # the smallest call: one step of one 192-tet StVK cantilever through
        # integrate with host buffers, as the reference's host code drives it
        {"name": "cantilever", "kind": "cantilever", "nx": 8, "ny": 2, "nz": 2, "copies": 1, "steps": 1},
        # thousands of small scenes stepped together on the device
        {"name": "cantilever_batch", "kind": "cantilever", "nx": 8, "ny": 2, "nz": 2, "copies": 4096, "steps": 8},
        # the two-layer Neo-Hookean block (98 k tets), resident stepper
        {"name": "block", "kind": "block", "nx": 64, "ny": 16, "nz": 16, "layers": 2, "fp64": False, "steps": 4},
        # the three-layer block of the benchmark (393 k tets)
        {"name": "block_large", "kind": "block", "nx": 64, "ny": 32, "nz": 32, "layers": 3, "fp64": False,
         "steps": 4},
        # a ragged block in FP64, the reference's own precision
        {"name": "block_fp64", "kind": "block", "nx": 37, "ny": 13, "nz": 11, "layers": 2, "fp64": True, "steps": 2},
        # a batch of uneven Neo-Hookean scenes (2 k to 40 k tets each) merged into one mesh
        {"name": "scene_batch", "kind": "batch", "scenes": 64, "tmin": 2000, "tmax": 40000, "steps": 4},
        # boxes dropped on a plane and spheres: contacts found on the device every step
        {"name": "drop", "kind": "drop", "boxes": 32, "cubes": 12, "coloring": True, "steps": 4},
        # the drop of one damped cube as simulate3D runs it: finders, layers by
        # strain rate rebuilt every step, host contact list, host buffers
        {"name": "drop_host", "kind": "drop_host", "nx": 11, "ny": 9, "nz": 7, "steps": 1},
        # a step solved to a residual with the stop rules on
        {"name": "to_residual", "kind": "residual", "nx": 32, "ny": 12, "nz": 12, "layers": 2, "pcg": False,
         "until": 1e-3},
        # the same on the benchmark's block with the PCG in the layer solve
        {"name": "to_residual_pcg", "kind": "residual", "nx": 64, "ny": 32, "nz": 32, "layers": 3, "pcg": True,
         "until": 1e-4},
        # steps with the learned warm start's network in the coarse layer
        {"name": "learned_step", "kind": "learned", "nx": 48, "ny": 24, "nz": 24, "steps": 2},
        # one batch of the warm start's training: loss and gradient
        {"name": "warm_start_fit", "kind": "fit", "rows": 4096},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["cantilever", "cantilever", "block", "block", "block", "batch", "drop", "drop_host", "residual",
                       "learned", "fit"])
    if kind == "cantilever":
        return {"kind": kind, "nx": rng.randint(4, 12), "ny": rng.randint(1, 3), "nz": rng.randint(1, 3),
                "copies": rng.choice([1, log_int(2, 2048)]), "steps": rng.randint(1, 8)}
    if kind == "block":
        fp64 = rng.random() < 0.25
        return {"kind": kind, "nx": log_int(12, 32 if fp64 else 64), "ny": log_int(6, 16 if fp64 else 32),
                "nz": log_int(6, 16 if fp64 else 32), "layers": rng.choice([2, 3]), "fp64": fp64,
                "steps": rng.randint(1, 4)}
    if kind == "batch":
        tmin = log_int(500, 4000)
        return {"kind": kind, "scenes": log_int(4, 64), "tmin": tmin, "tmax": tmin * rng.randint(2, 10),
                "steps": rng.randint(1, 4)}
    if kind == "drop":
        return {"kind": kind, "boxes": log_int(2, 32), "cubes": rng.randint(4, 12), "coloring": rng.random() < 0.6,
                "steps": rng.randint(1, 4)}
    if kind == "drop_host":
        return {"kind": kind, "nx": rng.randint(4, 14), "ny": rng.randint(4, 12), "nz": rng.randint(3, 10), "steps": 1}
    if kind == "residual":
        pcg = rng.random() < 0.6
        return {"kind": kind, "nx": log_int(12, 48 if pcg else 28), "ny": log_int(6, 24 if pcg else 12),
                "nz": log_int(6, 24 if pcg else 12), "layers": rng.choice([2, 3]), "pcg": pcg,
                "until": 1e-4 if pcg else 1e-3}
    if kind == "learned":
        return {"kind": kind, "nx": rng.randint(24, 48), "ny": rng.randint(12, 24), "nz": rng.randint(12, 24),
                "steps": rng.randint(1, 2)}
    return {"kind": kind, "rows": log_int(100, 4096)}


# ---------------------------------------------------------------------------
# Scenes: the mesh, its layers and the integrator settings.  They do not
# depend on the seed, so the host-side mesh generation runs once per size.

@lru_cache(maxsize=8)
def _scene(key):
    c = dict(key)
    if c["kind"] == "cantilever":
        one = scenes.config1()
        V, T, _ = scenes.generate_beam(c["nx"], c["ny"], c["nz"], 0.1)
        n, k = V.shape[0], np.arange(c["copies"])
        off = np.stack([np.zeros(k.size), 0.5 * (k % 64), 0.5 * (k // 64)], 1)
        V = (V[None] + off[:, None]).reshape(-1, 3)
        T = (T[None].astype(np.int64) + (n * k)[:, None, None]).reshape(-1, 4).astype(np.int32)
        mu, lam = to_lame(0.3, 1e5)
        m = Mesh3D.from_arrays(V, T, mu, lam, rho=1000.0, alpha1=0.0, energy_type=MLX_ENERGY_STVK_VOIGT)
        m.pin(np.nonzero(np.isclose(V[:, 0], 0.0))[0] + 1)
        one.mesh, one.custom_sets = m, np.zeros((m.T, 1), np.int32, order="F")
        return one
    if c["kind"] in ("block", "residual", "learned"):
        if c.get("layers", 3) == 2:
            return scenes.config2(nx=c["nx"], ny=c["ny"], nz=c["nz"])
        return scenes.config5(nx=c["nx"], ny=c["ny"], nz=c["nz"])
    if c["kind"] == "batch":
        return scenes.config3(n_scenes=c["scenes"], tmin=c["tmin"], tmax=c["tmax"])
    if c["kind"] == "drop":
        return scenes.config4(n_boxes=c["boxes"], cubes=c["cubes"], n_spheres=max(1, c["boxes"] // 8),
                              contact_coloring=c["coloring"])
    V, T, _ = scenes.generate_beam(c["nx"], c["ny"], c["nz"], 0.1)
    mu, lam = to_lame(0.3, 5e5)
    m = Mesh3D.from_arrays(V, T, mu, lam, rho=1000.0, alpha1=1e-3, energy_type=MLX_ENERGY_STVK_VOIGT)
    sc = scenes.Scene("drop_host", m, 1.0 / 120.0, 1, [50, 25, 0], [1, 4, 10])
    sc.contact_finders = [PlaneContactFinder3D([0.0, 0.0, 1.0], [0.0, 0.0, 0.0]),
                          SphereContactFinder(0.3, [0.05 * c["nx"], 0.05 * c["ny"], -0.2])]
    sc.settings["contactResistance"] = 0.9
    return sc


def _scene_of(case):
    return _scene(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "pcg", "until"))))


def _integrator(sc, precision):
    integ = XpbdLayer3D()
    integ.Gravity = sc.gravity
    integ.setLayers(sc.layers)
    integ.iterations = list(sc.iterations)
    integ.customRigidSets = sc.custom_sets
    integ.precision = precision
    integ.contactResistance = sc.settings.get("contactResistance", integ.contactResistance)
    integ.contactColoring = bool(sc.settings.get("contactColoring", False))
    return integ


@lru_cache(maxsize=8)
def _layers_of(sc_id):
    sc = _BY_ID[sc_id]
    sets = sc.custom_sets
    return find_boundary_vertices(sc.mesh, sets, [int(sets[:, k].max(initial=0)) for k in range(sets.shape[1])])


_BY_ID = {}


def _layer_set(sc):
    _BY_ID[id(sc)] = sc
    return _layers_of(id(sc))


def _start(case, sc, seed):
    """Positions and velocities in mid-motion: the mesh a little deformed, and
    for the drops every body just touching what lies under it."""
    rng = np.random.default_rng(seed)
    m = sc.mesh
    p, v = m.p.copy(), rng.normal(0.0, 0.05, 3 * m.N)
    if case["kind"] in ("residual", "learned"):
        # the step after a velocity impulse on a patch of the top surface
        V = p.reshape(-1, 3)
        top = np.nonzero(np.isclose(V[:, 2], V[:, 2].max()))[0]
        at = V[top[rng.integers(len(top))]]
        patch = top[np.linalg.norm(V[top, :2] - at[:2], axis=1) < 0.4]
        v[:] = 0.0
        v.reshape(-1, 3)[patch] = rng.normal(0.0, 0.5, (patch.size, 3)) + np.array([0.0, 0.0, -2.0])
    else:
        p += rng.normal(0.0, 5e-4, 3 * m.N)
    if case["kind"] == "drop":
        spheres = [f for f in sc.contact_finders if f.radius > 0]
        V = p.reshape(-1, 3)
        offs = getattr(m, "part_vertex_offsets")
        for a, b in zip(offs[:-1], offs[1:]):
            c = V[a:b].mean(0)
            under = [f.center[2] + f.radius for f in spheres if np.linalg.norm(f.center[:2] - c[:2]) < 0.5]
            V[a:b, 2] += (max(under) if under else 0.0) - 0.01 - V[a:b, 2].min()
        v.reshape(-1, 3)[:, 2] -= 1.0
    if case["kind"] == "drop_host":
        V = p.reshape(-1, 3)
        V[:, 2] += 0.1 - 0.01 - V[:, 2].min()
        v.reshape(-1, 3)[:, 2] -= 1.0
    v[m.pinnedDOFs - 1] = 0.0
    return p, v


def prepare(case, seed):
    if case["kind"] == "fit":
        rng = np.random.default_rng(seed)
        net = Mlp(44, 8, n_hidden=128, n_hidden_layers=3, max_batch=4096, seed=1)
        x = rng.normal(size=(case["rows"], 44)).astype(np.float32)
        y = np.tanh(x[:, :8] + 0.5 * x[:, 8:16]).astype(np.float32)
        return {"case": case, "net": net, "x": x, "y": y}
    sc = _scene_of(case)
    p, v = _start(case, sc, seed)
    fp64 = bool(case.get("fp64", False))
    st = {"case": case, "sc": sc, "p0": p, "v0": v, "dtype": np.float64 if fp64 else np.float32}
    integ = st["integ"] = _integrator(sc, MLX_FP64 if fp64 else MLX_FP32)
    if case["kind"] in ("drop_host", "residual") or (case["kind"] == "cantilever" and case["copies"] == 1):
        # the host-buffer path: a mesh object of this state's own
        m = st["mesh"] = Mesh3D.__new__(Mesh3D)
        m.__dict__.update(sc.mesh.__dict__)
        m.p, m.v = p.copy(), v.copy()
        st["cache"], st["frame"] = StepCache(), 0
        solver = st["solver"] = integ.solver(m)
        if case["kind"] == "residual":
            integ.computeResiduals = True
            integ.hangingStop = 4000
            if case["pcg"]:
                solver.layer_pcg()
        return st
    solver = st["solver"] = Solver(sc.mesh, precision=integ.precision)
    sim = st["sim"] = ResidentSim(solver, integ, _layer_set(sc), sc.h, p, v)
    if case["kind"] == "drop":
        sim.set_obstacles(sc.contact_finders)
    if case["kind"] == "learned":
        net, fn, on, _ = load_warm_start()
        sim.warm_start(mode=1, net=net, feature_norm=fn, output_norm=on)
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "fit":
        loss, grad = st["net"].loss_grad(st["x"], st["y"])
        return {"loss": np.float32(loss), "grad": grad}
    ft = st["dtype"]
    if "sim" in st:
        st["sim"].step(case["steps"])
        p, v = st["sim"].state()
        return {"p": p.astype(ft), "v": v.astype(ft)}
    m, integ, cache = st["mesh"], st["integ"], st["cache"]
    if case["kind"] == "residual":
        # every pass solves the same step to the residual
        m.p, m.v = st["p0"], st["v0"]
        integ.runUntilResSmallerThan = case["until"]
        out = integ.integrate(m, st["sc"].h, ContactSet(), cache, 1)
        res = np.zeros(integ.hangingStop + 96)  # one residual per iteration, as many as the solve took
        res[:cache.residualArray.size] = cache.residualArray
        return {"p": m.p.astype(ft), "v": m.v.astype(ft), "residuals": res, "iterations": int(out["iterations"])}
    contacts = ContactSet()
    for _ in range(case["steps"]):
        st["frame"] += 1
        if case["kind"] == "drop_host":
            contacts = find_contacts(st["solver"], st["sc"].contact_finders, m.p)
        integ.integrate(m, st["sc"].h, contacts, cache, st["frame"])
    return {"p": m.p.astype(ft), "v": m.v.astype(ft), "contacts": int(contacts.vertex_ids.size)}


def work(case):
    """One pass: per step each tet's rest data and each vertex's state once,
    the arithmetic of every projection; the state out once."""
    if case["kind"] == "fit":
        n = 44 * 128 + 2 * 128 * 128 + 128 * 8
        return {"bytes": 4.0 * (case["rows"] * 52 + 2 * n), "flops": 6.0 * case["rows"] * n}
    sc = _scene_of(case)
    m, steps = sc.mesh, case.get("steps", 1)
    word = 8 if case.get("fp64") else 4
    nh = m.energy_type == MLX_ENERGY_NEOHOOKEAN
    rest = 16 + word * (9 + (2 if nh else 3))
    its = 0.0
    for k, layer in enumerate(sc.layers):
        share = 1.0
        if sc.custom_sets is not None:
            share = float(np.mean(sc.custom_sets[:, sorted(set(sc.layers)).index(layer)] == 0))
        elif layer:
            share = 1.0 - layer / 100.0
        its += share * sc.iterations[k]
    if case["kind"] == "residual":
        its += 60.0 if not case["pcg"] else 100.0  # a solve takes some tens of iterations at least
    return {"bytes": float(steps * (m.T * rest + 4.0 * m.N * 4 * word)) + 48.0 * m.N,
            "flops": steps * its * m.T * (430.0 if nh else 520.0)}


# ---------------------------------------------------------------------------
# The step in 64 bits with plain torch, for the cases without contacts and
# without data-dependent iteration counts (those end on a comparison that the
# two precisions take at different iterations), and without a network.

def exact(case, seed):
    if case["kind"] == "fit":
        return _exact_fit(case, seed)
    if case["kind"] not in ("cantilever", "block", "batch"):
        return None
    sc = _scene_of(case)
    p, v = _start(case, sc, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, u = _exact_steps(sc, _layer_set(sc), p, v, case["steps"], dev)
    out = {"p": x.reshape(-1).cpu().numpy(), "v": u.reshape(-1).cpu().numpy()}
    return out


def _exact_fit(case, seed):
    rng = np.random.default_rng(seed)
    x = torch.from_numpy(rng.normal(size=(case["rows"], 44)).astype(np.float32))
    y = torch.tanh(x[:, :8] + 0.5 * x[:, 8:16]).double()
    net = Mlp(44, 8, n_hidden=128, n_hidden_layers=3, max_batch=128, seed=1)  # for its starting weights only
    flat, at, leaves, h = torch.from_numpy(net.get_params()).double(), 0, [], x.double()
    shapes = net.layer_shapes()
    for k, (no, ni) in enumerate(shapes):
        W = flat[at:at + no * ni].reshape(no, ni).clone().requires_grad_()
        b = flat[at + no * ni:at + no * ni + no].clone().requires_grad_()
        at += no * ni + no
        leaves += [W, b]
        h = h @ W.T + b
        if k + 1 < len(shapes):
            h = torch.nn.functional.gelu(h, approximate="tanh")
    loss = ((h - y) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "grad": torch.cat([t.grad.reshape(-1) for t in leaves]).numpy()}


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _rotation(w, h):
    mag = w.norm(dim=-1)
    u = torch.nan_to_num(w / mag[:, None])
    K = torch.zeros(w.shape[0], 3, 3, dtype=w.dtype, device=w.device)
    K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -u[:, 2], u[:, 1], -u[:, 0]
    K = K - K.transpose(1, 2)
    a = (h * mag)[:, None, None]
    return torch.eye(3, dtype=w.dtype, device=w.device) + torch.sin(a) * K + (1 - torch.cos(a)) * (K @ K)


class _Tets:
    """The tets of one colour of one layer."""

    def __init__(self, m, ids, minv, dev):
        g = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        self.ids = g(ids)
        self.v = g(np.asarray(m.t, np.int64)[ids] - 1)
        self.G = g(m.DmInv[ids].reshape(-1, 3, 3)).transpose(1, 2).contiguous()  # rows of DmInv
        self.m = minv[self.v][..., None]
        self.vol, self.mu, self.la = g(m.elV[ids]), g(m.mu[ids]), g(m.lam[ids])
        self.D = torch.cat([-self.G.sum(1, keepdim=True), self.G], 1)  # d F / d x_a, (n, 4, 3)


def _project_nh(q, x, lam, h):
    X = x[q.v]
    F = X.transpose(1, 2) @ q.D
    f0, f1, f2 = F.unbind(-1)
    cof = torch.stack([torch.linalg.cross(f1, f2), torch.linalg.cross(f2, f0), torch.linalg.cross(f0, f1)], -1)
    J = (f0 * cof[..., 0]).sum(-1)
    B = (F * F).sum((1, 2)) + J * J - 4 * J
    CD = B.clamp_min(0).sqrt()
    P = torch.where(CD > 1e-12, 1 / CD, torch.zeros_like(CD))[:, None, None] * (F + (J - 2)[:, None, None] * cof)
    gD, gH = q.D @ P.transpose(1, 2), q.D @ cof.transpose(1, 2)  # (n, 4, 3)
    has = q.la > q.mu
    aD = 1 / (q.vol * q.mu) / h ** 2
    aH = torch.where(has, 1 / (q.vol * (q.la - q.mu)) / h ** 2, torch.zeros_like(aD))
    a11, a22 = (q.m * gD * gD).sum((1, 2)) + aD, (q.m * gH * gH).sum((1, 2)) + aH
    a12 = (q.m * gD * gH).sum((1, 2))
    l0, l1 = lam[0, q.ids], lam[1, q.ids]
    b1, b2 = -CD - aD * l0, -(J - 1) - aH * l1
    det = a11 * a22 - a12 * a12
    d0 = torch.where(has, (b1 * a22 - a12 * b2) / det, b1 / a11)
    d1 = torch.where(has, (a11 * b2 - a12 * b1) / det, torch.zeros_like(b1))
    lam[0, q.ids], lam[1, q.ids] = l0 + d0, l1 + d1
    x[q.v] = X + q.m * (d0[:, None, None] * gD + d1[:, None, None] * gH)


def _project_stvk(q, x, lam, h):
    X = x[q.v]
    f = -(X.transpose(1, 2) @ q.D).transpose(1, 2)  # rows f_i
    d = -q.D
    FF, W = f @ f.transpose(1, 2), d.transpose(1, 2) @ (q.m * d)
    vol, eye = q.vol, torch.eye(3, dtype=x.dtype, device=x.device)
    C = vol[:, None, None] * 0.5 * (FF - eye)
    K = torch.diag_embed((4 * q.mu)[:, None].expand(-1, 3)) + q.la[:, None, None]
    aT, aS = torch.linalg.inv(K) / h ** 2, 1 / (2 * q.mu) / h ** 2
    l = lam[:, q.ids]
    A = (vol * vol)[:, None, None] * W * FF + aT
    b = -C.diagonal(dim1=1, dim2=2) - (aT @ l[:3].T[..., None])[..., 0]
    top = torch.linalg.solve(A, b)
    sh = []
    for k, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
        S = vol * vol * 0.25 * (W[:, i, i] * FF[:, j, j] + 2 * W[:, i, j] * FF[:, i, j] + W[:, j, j] * FF[:, i, i])
        sh.append((-C[:, i, j] - aS * l[3 + k]) / (S + aS))
    lam[:, q.ids] = l + torch.cat([top.T, torch.stack(sh)])
    L = torch.zeros_like(FF)
    for i in range(3):
        L[:, i, i] = top[:, i]
    for k, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
        L[:, i, j] = L[:, j, i] = 0.5 * sh[k]
    x[q.v] = X + q.m * vol[:, None, None] * ((d @ L) @ f)


class _Bodies:
    """The rigid bodies of one layer (cluster momentum, rotation, glue)."""

    def __init__(self, ids, nb, mass, x, u):
        self.ids, self.nb = ids, nb
        self.rv = torch.nonzero(ids > 0)[:, 0]
        self.b = ids[self.rv] - 1
        m = mass[self.rv][:, None]
        self.M = self.total(m)
        self.com, self.dot = self.total(m * x[self.rv]) / self.M, self.total(m * u[self.rv]) / self.M
        self.r = x[self.rv] - self.com[self.b]
        I = torch.eye(3, dtype=x.dtype, device=x.device) * _dot(self.r, self.r)[..., None]
        I = m[..., None] * (I - self.r[:, :, None] * self.r[:, None, :])
        self.I0 = self.total(I.reshape(-1, 9)).reshape(-1, 3, 3)
        L = self.total(m * torch.linalg.cross(self.r, u[self.rv] - self.dot[self.b]))
        self.omega = torch.linalg.solve(self.I0, L)
        self.R = torch.eye(3, dtype=x.dtype, device=x.device).expand(nb, 3, 3).clone()

    def total(self, a, b=None):
        return torch.zeros(self.nb, a.shape[1], dtype=a.dtype, device=a.device).index_add_(0, self.b if b is None else b, a)

    def turn(self, w, h):
        self.R = _rotation(w, h) @ self.R
        self.I = self.R @ self.I0 @ self.R.transpose(1, 2)

    def points(self):
        return (self.R[self.b] @ self.r[..., None])[..., 0] + self.com[self.b]


def _exact_steps(sc, ls, p, v, steps, dev):
    m, h = sc.mesh, sc.h
    g = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), device=dev).to(t)
    mass = g(m.mass).reshape(-1, 3)[:, 0]
    minv, x, u = 1 / mass, g(p).reshape(-1, 3).clone(), g(v).reshape(-1, 3).clone()
    pins = g(np.asarray(m.pinnedDOFs, np.int64) - 1, torch.int64)
    free = torch.ones(3 * m.N, dtype=torch.bool, device=dev)
    free[pins] = False
    pinx = x.reshape(-1)[pins].clone()
    project = _project_nh if m.energy_type == MLX_ENERGY_NEOHOOKEAN else _project_stvk
    columns = sorted(set(sc.layers))
    colour = np.asarray(m.elementColor)
    sweeps, bodies_of, glue_of = {}, {}, {}
    for layer in columns:
        k = columns.index(layer)
        el = np.asarray(ls.isElasticElement)[:, k] != 0
        sweeps[layer] = [_Tets(m, ids, minv, dev) for ids in
                         (np.nonzero(el & (colour == c))[0] for c in range(1, m.numColors + 1)) if ids.size]
        bodies_of[layer] = (g(ls.vertexRigidBody[:, k], torch.int64), int(ls.numRigids[k]))
        glue_of[layer] = g(np.nonzero(ls.isBoundaryVertex[:, k])[0], torch.int64)
    integ = XpbdLayer3D()
    bc, grav = integ.boundaryCompliance, sc.gravity
    for _ in range(steps):
        old = x.clone()
        fz = torch.zeros_like(x)
        fz[:, 2] = grav
        res = u + h * torch.where(free.reshape(-1, 3), fz, torch.zeros_like(fz))
        lam = torch.zeros(6, m.T, dtype=x.dtype, device=dev)
        for layer, its in zip(sc.layers, sc.iterations):
            ids, nb = bodies_of[layer]
            prev = x.clone()
            B = _Bodies(ids, nb, mass, x, res) if nb else None
            loose = ids == 0
            x[loose] += h * res[loose]
            res[loose] = 0
            if nb:
                B.com = B.com + h * B.dot
                B.turn(B.omega, h)
                step_R = B.R.clone()
                x[B.rv] = B.points()
                res[B.rv] = (B.R[B.b] @ res[B.rv][..., None])[..., 0] - (x[B.rv] - prev[B.rv]) / h
                gv = glue_of[layer]
                gb = ids[gv] - 1
                gr = torch.zeros_like(x)
                gr[B.rv] = B.r
                gr, lb = gr[gv], torch.zeros(gv.numel(), 1, dtype=x.dtype, device=dev)
            for _ in range(its):
                for q in sweeps[layer]:
                    project(q, x, lam, h)
                if nb and gv.numel():
                    r = (B.R[gb] @ gr[..., None])[..., 0]
                    to = r + B.com[gb] - x[gv]
                    C = to.norm(dim=-1, keepdim=True)
                    n = torch.nan_to_num(to / C)
                    ax = torch.linalg.cross(r, n)
                    w = 1 / B.M[gb] + _dot(ax, torch.linalg.solve(B.I[gb], ax))
                    dl = (-C - bc * lb) / (minv[gv][:, None] + w + bc)
                    lb = lb + dl
                    B.com = B.com + B.total(dl * n / B.M[gb], gb)
                    B.turn(torch.linalg.solve(B.I, B.total(torch.linalg.cross(r, dl * n / h), gb)), h)
                    x[gv] = (B.R[gb] @ gr[..., None])[..., 0] + B.com[gb]
                x.reshape(-1)[pins] = pinx
            if nb:
                x[B.rv] = B.points()
                dR = B.R @ step_R.transpose(1, 2)
                res[B.rv] = (dR[B.b] @ res[B.rv][..., None])[..., 0]
        u = (x - old) / h
    return x, u
