"""Timing cases of the library's public entry points.

Each case is a dict of plain values; ``prepare`` makes what a program has in
hand before the call (mesh, handle, inputs), ``run`` makes one pass through
the public entry points and returns everything it computes, ``exact`` gives
the same outputs in 64-bit torch, without this library's kernels, and
``work`` what the pass cannot do without.

Meshes are the repository's synthetic disks (``meshgen``); their host set-up
is kept per mesh, as a program that steps one mesh from many starts keeps it.
Start states are taken from the middle of a run, with the dial factor half
way: the cone an azimuthal director field pulls the sheet into (a gentle dome
for the other fields), with the set-up noise and seeded smooth modes on top,
moving at a seeded smooth velocity.
"""
from __future__ import annotations

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from morphoshell_b200 import (MS_PRECISION_FP64, MS_PRECISION_MIXED, Batch, GpuLoop, Mlp, Model, lib, meshgen,
                              warmstart)

DIAL0 = 0.52           # dial factor the start states are taken at
L2_BYTES = 126e6
TRI_FLOPS = 850        # per triangle-step: derivatives, energy gradient, contributions (fma = 2)
PRECISIONS = {"fp64": MS_PRECISION_FP64, "mixed": MS_PRECISION_MIXED}


def listed():
    return [
        # Main-loop stretches (dialling or waiting for equilibrium) between
        # two host decisions, from host state to host state: the smallest
        # test mesh, where a step is all latency; the 18k-triangle disk most
        # runs use, dialling and waiting; the 1.8M-triangle benchmark disk,
        # in both precisions.
        {"name": "step_disk100", "kind": "steps", "spacing": 0.1, "steps": 256, "precision": "fp64",
         "dialling": True, "check": False},
        {"name": "step_disk18k", "kind": "steps", "spacing": 0.02, "steps": 1000, "precision": "fp64",
         "dialling": True, "check": False},
        {"name": "wait_disk18k_mixed", "kind": "steps", "spacing": 0.02, "steps": 1000, "precision": "mixed",
         "dialling": False, "check": True},
        {"name": "step_disk1p8m", "kind": "steps", "spacing": 0.002, "steps": 300, "precision": "fp64",
         "dialling": True, "check": False},
        {"name": "step_disk1p8m_mixed", "kind": "steps", "spacing": 0.002, "steps": 300, "precision": "mixed",
         "dialling": True, "check": False},
        # One step through the one-call-per-function path, as the driver
        # takes it on equilibrium-check steps (147,922 triangles).
        {"name": "check_disk7", "kind": "functions", "spacing": 0.007},
        # The quantities of one output file, on a ragged mid-size mesh.
        {"name": "output_disk13", "kind": "outputs", "spacing": 0.013},
        # Forces for callers that own all device memory, near the largest
        # mesh that entry point takes.
        {"name": "forces_noalloc_disk12", "kind": "noalloc", "spacing": 0.012},
        # Batched ensembles: members of mixed sizes, and many programmed
        # fields on one small mesh (the warm start's training data).
        {"name": "ensemble8", "kind": "ensemble", "members": 8, "first": 0, "steps": 128, "precision": "fp64"},
        {"name": "fields64_disk40", "kind": "fields", "spacing": 0.04, "members": 64, "steps": 256,
         "precision": "fp64"},
        # The warm-start network: the prediction for one mesh's nodes, and
        # training epochs over a data set with a ragged last batch.
        {"name": "net_forward_9201", "kind": "net_forward", "rows": 9201, "width": 256, "hidden": 4},
        {"name": "net_train_100003", "kind": "net_train", "rows": 100003, "batch": 8192, "epochs": 3, "width": 256,
         "hidden": 4},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "functions", "outputs", "noalloc", "ensemble", "fields",
                       "net_forward", "net_train"])
    if kind == "steps":
        spacing = round(_log_uniform(rng, 0.002, 0.1), 5)
        room = 300 * 1.8e6 / (7.26 / spacing ** 2)
        dialling = rng.random() < 0.6
        return {"kind": kind, "spacing": spacing, "steps": int(max(1, min(room, _log_uniform(rng, 1, 1000)))),
                "precision": rng.choice(["fp64", "fp64", "mixed"]), "dialling": dialling,
                "check": not dialling and rng.random() < 0.7}
    if kind in ("functions", "outputs"):
        return {"kind": kind, "spacing": round(_log_uniform(rng, 0.005, 0.1), 5)}
    if kind == "noalloc":
        return {"kind": kind, "spacing": round(_log_uniform(rng, 0.0115, 0.1), 5)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(2, 8), "first": rng.randint(0, 200),
                "steps": int(_log_uniform(rng, 33, 128)), "precision": rng.choice(["fp64", "fp64", "mixed"])}
    if kind == "fields":
        return {"kind": kind, "spacing": round(rng.uniform(0.035, 0.1), 5), "members": rng.randint(3, 64),
                "steps": int(_log_uniform(rng, 64, 256)), "precision": rng.choice(["fp64", "fp64", "mixed"])}
    width = rng.choice([128, 256, 256, 256, 512])
    hidden = rng.randint(2, 5)
    if kind == "net_forward":
        return {"kind": kind, "rows": int(_log_uniform(rng, 376, 200000)), "width": width, "hidden": hidden}
    return {"kind": kind, "rows": int(_log_uniform(rng, 5000, 150000)), "batch": rng.choice([4096, 8192, 32768]),
            "epochs": rng.randint(1, 3), "width": width, "hidden": hidden}


# ---- inputs -----------------------------------------------------------------

_meshes: dict = {}


def _settings(**over):
    d = tempfile.mkdtemp(prefix="ms_cases_")
    path = os.path.join(d, "settings.txt")
    meshgen.write_settings(path, protocol=3, **over)
    return path


def _keep(key, make):
    """The last few set-ups: meshes are costly to generate and do not depend
    on the seed."""
    if key not in _meshes:
        while len(_meshes) >= 16:
            _meshes.pop(next(iter(_meshes)))
        _meshes[key] = make()
    return _meshes[key]


def _disk(spacing):
    """(Model, abar_info, bbar_info): the wavy azimuthal director with lambda
    1 -> 0.85 on fine meshes, the azimuthal one with 1 -> 0.9 on the others,
    as the named workloads have them."""
    def make():
        mesh = meshgen.disk_mesh(spacing, seed=1)
        if spacing < 0.01:
            info = meshgen.lce_abar_info(mesh, meshgen.wavy_azimuthal_director, 0.85)
        else:
            info = meshgen.lce_abar_info(mesh, meshgen.azimuthal_director, 0.9)
        bbar = np.zeros((mesh.num_tris, 3))
        return Model.from_arrays(_settings(), mesh.nodes, mesh.tris, info, bbar), info, bbar
    return _keep(("disk", spacing), make)


def _member(k):
    def make():
        mesh, info, bbar, over, _ = meshgen.ensemble_member(k)
        return Model.from_arrays(_settings(**over), mesh.nodes, mesh.tris, info, bbar), info
    return _keep(("member", k), make)


def _state(model, seed, lam_final=None):
    """Positions and velocities (3N, SoA) in the middle of a run.  With
    lam_final, near the cone whose circles are lambda and whose generators
    lambda^(-1/2) times their flat lengths, rounded at the tip."""
    rng = np.random.default_rng([seed, model.num_tris])
    x = model.dofs(1).reshape(3, -1).copy()
    X, Y = x[0].copy(), x[1].copy()
    r2 = X * X + Y * Y
    if lam_final is None:
        x[0] *= 1.0 + 0.02 * rng.uniform(0.5, 1.0)
        x[1] *= 1.0 - 0.02 * rng.uniform(0.5, 1.0)
        x[2] += 0.05 * rng.uniform(0.5, 1.0) * np.exp(-rng.uniform(1.5, 3.0) * r2)
    else:
        lam = (1.0 - DIAL0) + DIAL0 * lam_final
        x[:2] *= lam * (1.0 + 0.004 * rng.uniform(0.5, 1.0))
        x[2] += math.sqrt(1.0 / lam - lam * lam) * np.sqrt(r2 + 0.02 * rng.uniform(0.8, 1.2))
    speed = model.scalars.char_speed_scale
    v = np.zeros_like(x)
    for k in range(1, 4):
        p = rng.uniform(0.0, 2.0 * math.pi, 4)
        wave = np.sin(k * X + p[0]) * np.cos(k * Y + p[1])
        x[2] += 0.004 / k * rng.normal() * wave
        x[0] += 0.002 / k * np.sin(k * Y + p[2])
        v[0] += 1e-3 * speed / k * np.cos(k * X + p[3])
        v[1] += 1e-3 * speed / k * np.sin(k * Y + p[3])
        v[2] += 1e-2 * speed / k * wave
    return x.ravel(), v.ravel()


def _dials(s, steps):
    k = np.arange(steps, dtype=np.float64)
    return DIAL0 + s.dial_factors_to_hold_at_spacing * (k / float(s.timesteps_per_dial_phase))


def _features(rows, seed):
    """Rows of the network's data set: node features of random fields on one
    disk, and smooth displacements of the size equilibria have."""
    model, _, _ = _disk(0.04)
    xy = model.dofs(0).reshape(3, -1).T[:, :2]
    n = -(-rows // len(xy))
    x = np.concatenate([warmstart.node_features(xy, f) for f in warmstart.fields(n, seed)])[:rows]
    r, lam = x[:, 2], x[:, 13]
    t = np.stack([(lam - 1.0) * x[:, 0] * (1.0 + 0.2 * x[:, 11]), (lam - 1.0) * x[:, 1] * (1.0 + 0.2 * x[:, 12]),
                  0.4 * np.abs(lam - 1.0) * (1.0 - r * r) + 0.05 * x[:, 5]], 1)
    return np.ascontiguousarray(x, dtype=np.float32), np.ascontiguousarray(t, dtype=np.float32)


def _ptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "functions", "outputs"):
        model, info, bbar = _disk(case["spacing"])
        s = model.scalars
        g = GpuLoop(model, precision=PRECISIONS[case.get("precision", "fp64")], device=0)
        g.set_programmed(3, info, bbar, s.dial_factors_to_hold_at_spacing)
        g.do_dialling(DIAL0)
        x, v = _state(model, seed, info[0, 1])
        st = {"case": case, "loop": g, "x": x, "v": v, "dt": s.timestep,
              "damping": s.damping_factor_1 if case.get("dialling") else s.damping_factor_2}
        if kind == "steps" and case["dialling"]:
            st["dials"] = _dials(s, case["steps"])
        if kind == "outputs":
            g.upload(x, v)
        return st
    if kind == "noalloc":
        model, info, _ = _disk(case["spacing"])
        t = model.tables()
        x, _ = _state(model, seed, info[0, 1])
        T = model.num_tris
        abar = meshgen.lce_abar_comps(info, DIAL0)
        dev = {k: torch.from_numpy(np.ascontiguousarray(a)).cuda() for k, a in
               [("patch_ids", t["patch_ids"]), ("coef", t["deriv_coeffs"]), ("area", t["ref_area"]),
                ("thick", t["ref_thickness"]), ("shear", t["ref_shear_modulus"]), ("abar", abar),
                ("bbar", np.zeros((T, 3))), ("dofs", x)]}
        dev["forces"] = torch.empty_like(dev["dofs"])
        return {"case": case, "dev": dev, "N": model.num_nodes, "T": T, "nu": model.params.def_poisson_ratio,
                "gamma": model.params.bend_stiffening_scale_factor}
    if kind in ("ensemble", "fields"):
        models, infos = _instances(case, seed)
        b = Batch(models, precision=PRECISIONS[case["precision"]], device=0, abar_infos=infos)
        return {"case": case, "batch": b, "starts": [_state(m, seed + 1000 * i) for i, m in enumerate(models)]}
    net = Mlp(warmstart.N_FEATURES, width=case["width"], hidden_layers=case["hidden"], out_dim=3, seed=seed, device=0)
    x, t = _features(case["rows"], seed)
    st = {"case": case, "net": net, "x": x, "params": net.params(), "seed": seed}
    if kind == "net_train":
        net.set_data(x, t)
    return st


def _instances(case, seed):
    """Models and programmed fields of a batch case."""
    if case["kind"] == "ensemble":
        got = [_member(case["first"] + i) for i in range(case["members"])]
        return [m for m, _ in got], [a for _, a in got]
    model, _, _ = _disk(case["spacing"])
    cen = warmstart.centroids(model)
    infos = [warmstart.abar_info(cen, f) for f in warmstart.fields(case["members"], seed)]
    return [model] * case["members"], infos


# ---- one pass ---------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        g = state["loop"]
        g.upload(state["x"], state["v"])
        rep = g.step_n(case["steps"], state.get("dials"), state["dt"], state["damping"], check_last=case["check"])
        x, v = g.download()
        out = {"dofs": x, "velocities": v, "steps": rep.steps_done}
        if case["check"]:
            out.update(max_force=rep.equil.max_force, max_speed=rep.equil.max_speed,
                       max_force_node=rep.equil.max_force_node, max_speed_node=rep.equil.max_speed_node)
        return out
    if kind == "functions":
        # The driver's check step; intermediate results stay on the device.
        g, L = state["loop"], lib()
        g.upload(state["x"], state["v"])
        g._chk(L.ms_surface_derivs(g._h, None), "surface_derivs")
        g.do_dialling(DIAL0)
        g._chk(L.ms_deformation_forces(g._h, None, None), "deformation_forces")
        g.non_deformation_forces(state["damping"])
        g.impose_constraints()
        eq = g.is_at_equilibrium()
        g.advance_dynamics(state["dt"], state["damping"])
        x, v = g.download()
        return {"dofs": x, "velocities": v, "forces": g.forces(), "max_force": eq.max_force,
                "max_speed": eq.max_speed, "max_force_node": eq.max_force_node, "max_speed_node": eq.max_speed_node}
    if kind == "outputs":
        return state["loop"].output_quantities()
    if kind == "noalloc":
        d = state["dev"]
        err = ctypes.create_string_buffer(256)
        p = [ctypes.c_void_p(d[k].data_ptr()) for k in ("patch_ids", "coef", "area", "thick", "shear", "abar", "bbar")]
        rc = lib().ms_deformation_forces_noalloc(
            state["N"], state["T"], *p, state["nu"], state["gamma"], ctypes.c_void_p(d["dofs"].data_ptr()),
            ctypes.c_void_p(d["forces"].data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), err,
            256)
        if rc != 0:
            raise RuntimeError(err.value.decode())
        return d["forces"]
    if kind in ("ensemble", "fields"):
        b = state["batch"]
        for i, (x, v) in enumerate(state["starts"]):
            b.upload(i, x, v)
            b.set_start(i, DIAL0, False)
        b.run(case["steps"])
        got = [b.download(i) for i in range(b.n)]
        return {"dofs": np.concatenate([x for x, _ in got]), "velocities": np.concatenate([v for _, v in got])}
    net = state["net"]
    if kind == "net_forward":
        return net.forward(state["x"])
    net.set_params(state["params"])
    losses = net.train(case["epochs"], batch=case["batch"], lr=1e-3, seed=state["seed"])
    return {"losses": losses, "params": net.params()}


# ---- 64-bit values ------------------------------------------------------------

class _Shell:
    """The force-and-dynamics loop of one mesh in 64-bit torch: forces as the
    gradient of the elastic energy."""

    def __init__(self, model, info):
        dev = "cuda"
        t = model.tables()
        f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)
        self.ids = f(t["patch_ids"]).long()
        c = f(t["deriv_coeffs"])
        self.d1, self.d2 = c[:, :6].reshape(-1, 2, 3), c[:, 6:].reshape(-1, 6, 3)
        self.area, h, mu = f(t["ref_area"]), f(t["ref_thickness"]), f(t["ref_shear_modulus"])
        self.mass, self.fixed = f(t["node_mass"]), f(t["is_constrained"]).bool()
        self.boundary = f(t["is_boundary"]).bool()
        p = model.params
        self.nu = p.def_poisson_ratio
        self.ks, self.kb = 2 * h * mu / (1 - self.nu), mu * h ** 3 / (6 * (1 - self.nu))
        self.igmh = 1.0 / (p.bend_stiffening_scale_factor * mu * h)
        self.rho_hh = p.ref_density * p.min_ref_thickness ** 2
        self.info = f(info)
        self.N = model.num_nodes

    def metric(self, dial):
        ang, lf, nu = self.info[:, 0], self.info[:, 1], self.info[:, 2]
        lam = (1.0 - dial) + dial * lf
        p, l2 = lam ** (-2.0 * nu), lam * lam
        c, s = torch.cos(ang), torch.sin(ang)
        return l2 * c * c + p * s * s, (l2 - p) * c * s, p * c * c + l2 * s * s

    def surface(self, x):
        P = x[self.ids]                                   # [T, 6, 3]
        r1 = torch.bmm(self.d1, P[:, :3])                 # [T, 2, 3]
        r2 = torch.bmm(self.d2.transpose(1, 2), P)        # [T, 3, 3]: xx, xy, yy
        rx, ry = r1[:, 0], r1[:, 1]
        cr = torch.linalg.cross(rx, ry)
        n = cr / cr.norm(dim=1, keepdim=True)
        b = -(r2 * n[:, None, :]).sum(2)
        a = ((rx * rx).sum(1), (rx * ry).sum(1), (ry * ry).sum(1))
        return rx, ry, cr, a, (b[:, 0], b[:, 1], b[:, 2])

    def _form(self, ab, d):
        m00, m01 = ab[2] * d[0] - ab[1] * d[1], ab[2] * d[1] - ab[1] * d[2]
        m10, m11 = ab[0] * d[1] - ab[1] * d[0], ab[0] * d[2] - ab[1] * d[1]
        return (1 - self.nu) * (m00 * m00 + 2 * m01 * m10 + m11 * m11) + self.nu * (m00 + m11) ** 2

    def densities(self, ab, a, b):
        det = (ab[0] * ab[2] - ab[1] * ab[1]) ** -1.5
        ws = 0.5 * self.ks * det * self._form(ab, [p - q for p, q in zip(a, ab)])
        wb = 0.5 * self.kb * det * self._form(ab, b)
        return ws, wb * (1 + wb * self.igmh)

    def forces(self, x, ab):
        x = x.detach().requires_grad_(True)
        _, _, _, a, b = self.surface(x)
        ws, wb = self.densities(ab, a, b)
        (g,) = torch.autograd.grad((self.area * (ws + wb)).sum(), x)
        return -g

    def step(self, x, v, ab, dt, damping):
        F = self.forces(x, ab) - (damping / self.rho_hh) * self.mass[:, None] * v
        F[self.fixed] = 0.0
        v1 = v + dt * F / self.mass[:, None]
        return x + dt * v1, v1, F


def _nodes(a):
    return torch.from_numpy(a.reshape(3, -1).T.copy()).cuda()


def _flat(t):
    return t.T.contiguous().reshape(-1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "net_train":
        return None  # the order of the shuffled rows is the library's own
    if kind == "net_forward":
        net = Mlp(warmstart.N_FEATURES, width=case["width"], hidden_layers=case["hidden"], out_dim=3, seed=seed,
                  device=0)
        p = torch.from_numpy(net.params().astype(np.float64)).cuda()
        x, _ = _features(case["rows"], seed)
        h = torch.zeros(case["rows"], net.in_pad, dtype=torch.float64, device="cuda")
        h[:, :net.in_dim] = torch.from_numpy(x).cuda()
        lay = net.layers()
        for i, (off, n, k, _) in enumerate(lay):
            z = h @ p[off:off + n * k].reshape(n, k).T + p[off + n * k:off + n * k + n]
            h = z if i == len(lay) - 1 else z * torch.sigmoid(z)
        return h.cpu().numpy()
    if kind in ("ensemble", "fields"):
        models, infos = _instances(case, seed)
        xs, vs = [], []
        for i, (m, a) in enumerate(zip(models, infos)):
            s = m.scalars
            x, v = (_nodes(q) for q in _state(m, seed + 1000 * i))
            shell = _Shell(m, a)
            # The phase counter resumes inside the phase the start's dial
            # factor falls in; the first step dials to that factor itself.
            k0 = int(math.fmod(DIAL0, s.dial_factors_to_hold_at_spacing) * s.timesteps_per_dial_phase)
            for k in range(case["steps"]):
                dial = DIAL0 if k == 0 else DIAL0 + s.dial_factors_to_hold_at_spacing * (
                    (k0 + k) / s.timesteps_per_dial_phase)
                x, v, _ = shell.step(x, v, shell.metric(dial), s.timestep, s.damping_factor_1)
            xs.append(_flat(x))
            vs.append(_flat(v))
        return {"dofs": np.concatenate(xs), "velocities": np.concatenate(vs)}
    model, info, _ = _disk(case["spacing"])
    s = model.scalars
    x, v = (_nodes(q) for q in _state(model, seed, info[0, 1]))
    shell = _Shell(model, info)
    if kind == "noalloc":
        return _flat(shell.forces(x, shell.metric(DIAL0)))
    if kind == "outputs":
        ab = shell.metric(DIAL0)
        rx, ry, cr, a, b = shell.surface(x)
        ws, wb = shell.densities(ab, a, b)
        det = a[0] * a[2] - a[1] * a[1]
        curv = torch.stack([(b[0] * b[2] - b[1] * b[1]) / det,
                            0.5 * (a[2] * b[0] - 2 * a[1] * b[1] + a[0] * b[2]) / det], 1)
        d = [p - q for p, q in zip(a, ab)]
        x00, x01 = (a[2] * d[0] - a[1] * d[1]) / det, (a[2] * d[1] - a[1] * d[2]) / det
        x10, x11 = (a[0] * d[1] - a[1] * d[0]) / det, (a[0] * d[2] - a[1] * d[1]) / det
        strain = (0.125 * (x00 * x00 + 2 * x01 * x10 + x11 * x11)).sqrt()
        P = x[shell.ids[:, :3]]
        deficit = (2.0 - shell.boundary.double()) * math.pi
        for i in range(3):
            e, f = P[:, (i + 1) % 3] - P[:, i], P[:, (i + 2) % 3] - P[:, i]
            ang = torch.acos((e * f).sum(1) / (e.norm(dim=1) * f.norm(dim=1)))
            deficit.index_add_(0, shell.ids[:, i], -ang)
        kin = 0.5 * (shell.mass[:, None] * v * v).sum()
        return {"curvatures": curv.cpu().numpy(), "energy_densities": torch.stack([ws, wb], 1).cpu().numpy(),
                "strains": strain.cpu().numpy(), "stresses": None, "angle_deficits": deficit.cpu().numpy(),
                "energies": torch.stack([(shell.area * ws).sum(), (shell.area * wb).sum(), kin]).cpu().numpy()}
    if kind == "functions":
        x1, v1, F = shell.step(x, v, shell.metric(DIAL0), s.timestep, s.damping_factor_2)
        return {"dofs": _flat(x1), "velocities": _flat(v1), "forces": _flat(F),
                "max_force": float(F.norm(dim=1).max()), "max_speed": float(v.norm(dim=1).max()),
                "max_force_node": None, "max_speed_node": None}
    dials = _dials(s, case["steps"]) if case["dialling"] else None
    damping = s.damping_factor_1 if case["dialling"] else s.damping_factor_2
    held = None if case["dialling"] else shell.metric(DIAL0)
    for k in range(case["steps"]):
        v0 = v
        x, v, F = shell.step(x, v, shell.metric(float(dials[k])) if held is None else held, s.timestep, damping)
    out = {"dofs": _flat(x), "velocities": _flat(v), "steps": None}
    if case["check"]:
        out.update(max_force=float(F.norm(dim=1).max()), max_speed=float(v0.norm(dim=1).max()), max_force_node=None,
                   max_speed_node=None)
    return out


# ---- what a pass cannot do without ----------------------------------------------

def _table_bytes(T, precision):
    """Patch ids, derivative weights, programmed columns and area of T triangles."""
    return T * (24 + (96 if precision == "mixed" else 192) + 24 + 8)


def _loop_work(T, steps, precision):
    """A mesh whose tables and state stay on chip is read once, a larger one
    once a step; the state goes in and out by the host."""
    N = T / 2
    once = _table_bytes(T, precision) + 104 * N
    moved = once * steps if once > L2_BYTES else once
    return {"bytes": moved + 96 * N, "flops": float(TRI_FLOPS) * T * steps}


def work(case):
    kind = case["kind"]
    if kind == "net_forward":
        per_row = warmstart.network_flops_per_row(warmstart.N_FEATURES, case["width"], case["hidden"])
        return {"bytes": case["rows"] * 4 * (warmstart.N_FEATURES + 3), "flops": per_row * case["rows"]}
    if kind == "net_train":
        per_row = warmstart.network_flops_per_row(warmstart.N_FEATURES, case["width"], case["hidden"])
        rows = case["rows"] * case["epochs"]
        return {"bytes": rows * 4 * (warmstart.N_FEATURES + 3), "flops": 3.0 * per_row * rows}
    if kind in ("ensemble", "fields"):
        if kind == "ensemble":
            T = sum(_disk_tris(meshgen.ensemble_params(case["first"] + i)["spacing"]) for i in range(case["members"]))
        else:
            T = case["members"] * _disk_tris(case["spacing"])
        return _loop_work(T, case["steps"], case["precision"])
    T = _disk_tris(case["spacing"])
    if kind == "steps":
        return _loop_work(T, case["steps"], case["precision"])
    if kind == "outputs":
        return {"bytes": _table_bytes(T, "fp64") + 13 * 8 * T + (48 + 8) * T / 2, "flops": 1200.0 * T}
    if kind == "functions":
        return {"bytes": _table_bytes(T, "fp64") + (104 + 24) * T / 2, "flops": float(TRI_FLOPS) * T}
    return {"bytes": T * (24 + 192 + 24 + 48) + 48 * T / 2, "flops": float(TRI_FLOPS) * T}


def _disk_tris(spacing):
    """Triangles of a disk of this spacing, to a few per cent."""
    return 7.26 / spacing ** 2
