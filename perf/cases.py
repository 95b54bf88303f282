"""Performance cases: the calls that users of this package make, over the sizes they make them at.

Kinds of case (all through ``shape_atrophy_gb300.api`` with host arrays, as its callers pass them):

* ``frame2d`` / ``frame3d`` -- forward solve and objective of the frame model (K-preconditioned CG with the dense
  RKHS matrix) on a strip / an icosphere shell;
* ``layered2d`` / ``layered3d`` -- forward solve, with or without the objective, of the layered model (block-Jacobi
  PCG) on an annulus / an icosphere shell, FP64 or mixed precision, one or several parameter columns;
* ``varifold2d`` / ``varifold3d`` -- the varifold objective of a given shape, alone or with its node gradient;
* ``adjoint2d`` / ``adjoint3d`` -- objective and its gradient with respect to every parameter (layered model);
* ``serve`` -- a batch of layered solves submitted at once to the continuous-batching server.

``exact`` restates the model with element-wise torch operations in 64 bits: converged conjugate gradients (or a
dense factorisation for the frame model's velocity) in place of the package's solvers, automatic differentiation in
place of its adjoint, all pairs of the varifold sums.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from shape_atrophy_gb300 import api, mesh


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a quick look at the frame model on a coarse strip: the smallest solve, launches and latency count
        dict(name="frame_strip_coarse", kind="frame2d", ang=21, lyr=7, steps=5, order=3),
        # the reference's demonstration strip (3131 nodes), the first steps of its run
        dict(name="frame_strip_demo", kind="frame2d", ang=101, lyr=31, steps=8, order=3),
        # the frame model in 3D, a small closed shell
        dict(name="frame_shell", kind="frame3d", level=3, lyr=4, steps=6, order=1),
        # the layered 2D annulus over its whole run: small systems, hundreds of iterations per step
        dict(name="annulus", kind="layered2d", ang=256, lyr=16, steps=50, materials=4, precision="fp64", columns=1,
             objective=True, tol=1e-11),
        # the layered 3D shell (92178 nodes, 491520 tetrahedra) with its objective: the ordinary large solve
        dict(name="shell", kind="layered3d", level=5, lyr=9, steps=10, precision="fp64", columns=1, objective=True,
             tol=1e-11),
        # the same in mixed precision
        dict(name="shell_mixed", kind="layered3d", level=5, lyr=9, steps=10, precision="mixed", columns=1,
             objective=True, tol=1e-11),
        # a finer surface (204810 nodes): a trajectory only, as a caller of deformation asks for it
        dict(name="shell_fine", kind="layered3d", level=6, lyr=5, steps=3, precision="fp64", columns=1,
             objective=False, tol=1e-11),
        # objective and node gradient of a closed curve: one evaluation inside an optimiser's line search
        dict(name="varifold_curve_gradient", kind="varifold2d", ang=256, lyr=16, cen="G", dir="B", width=0.1,
             grad=True, precision="fp64"),
        # the objective of a fine surface against a target of the same size
        dict(name="varifold_surface", kind="varifold3d", level=5, lyr=2, cen="M", dir="B", width=0.08, grad=False,
             precision="fp64"),
        # objective and gradient of a surface, the other kernels
        dict(name="varifold_surface_gradient", kind="varifold3d", level=4, lyr=3, cen="C", dir="O", width=0.15,
             grad=True, precision="fp64"),
        # all gradients of a small shell problem at once
        dict(name="adjoint_shell", kind="adjoint3d", level=3, lyr=5, steps=5, tol=1e-12),
        # a batch of requests, 2D and 3D, of several sizes, served together
        dict(name="serve_batch", kind="serve", requests=12, steps=8, precision="fp64", tol=1e-11),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame2d", "frame3d", "layered2d", "layered2d", "layered3d", "layered3d", "layered3d",
                       "varifold2d", "varifold3d", "varifold3d", "adjoint2d", "adjoint3d", "serve"])
    tol = 10.0 ** -rng.uniform(11.0, 12.0)
    if kind == "frame2d":
        lyr = rng.randint(5, 31)
        return dict(kind=kind, ang=_log_int(rng, 15, 101), lyr=lyr, steps=rng.randint(2, 8), order=rng.randint(1, 4))
    if kind == "frame3d":
        level = rng.choice([2, 2, 3])
        return dict(kind=kind, level=level, lyr=rng.randint(3, 7 if level == 2 else 4), steps=rng.randint(2, 6),
                    order=rng.randint(0, 4))
    if kind == "layered2d":
        lyr = rng.randint(6, 24)
        return dict(kind=kind, ang=_log_int(rng, 48, 512), lyr=lyr, steps=rng.randint(5, 40),
                    materials=rng.randint(2, 5), precision=rng.choice(["fp64", "fp64", "mixed"]),
                    columns=rng.choice([1, 1, 3]), objective=rng.random() < 0.7, tol=tol)
    if kind == "layered3d":
        level = rng.choice([2, 3, 4, 4, 5])
        return dict(kind=kind, level=level, lyr=rng.randint(3, 13 if level < 5 else 9), steps=rng.randint(3, 10),
                    precision=rng.choice(["fp64", "mixed"]), columns=1, objective=rng.random() < 0.5, tol=tol)
    if kind == "varifold2d":
        return dict(kind=kind, ang=_log_int(rng, 40, 2500), lyr=rng.randint(3, 16), cen=rng.choice(["G", "C", "M"]),
                    dir=rng.choice(["B", "L", "O", "U"]), width=rng.uniform(0.05, 0.3), grad=rng.random() < 0.6,
                    precision="fp64")
    if kind == "varifold3d":
        grad = rng.random() < 0.5
        level = rng.choice([2, 3, 4]) if grad else rng.choice([2, 3, 4, 5])
        return dict(kind=kind, level=level, lyr=rng.randint(2, 4), cen=rng.choice(["G", "C", "M"]),
                    dir=rng.choice(["B", "L", "O", "U"]), width=rng.uniform(0.06, 0.3), grad=grad,
                    precision="fp64" if grad else rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "adjoint2d":
        return dict(kind=kind, ang=_log_int(rng, 40, 256), lyr=rng.randint(6, 16), steps=rng.randint(3, 10), tol=1e-12)
    if kind == "adjoint3d":
        return dict(kind=kind, level=rng.choice([2, 3]), lyr=rng.randint(3, 7), steps=rng.randint(2, 6), tol=1e-12)
    return dict(kind=kind, requests=rng.randint(3, 12), steps=rng.randint(3, 8),
                precision=rng.choice(["fp64", "mixed"]), tol=tol)


# ---------------------------------------------------------------------------
# inputs: a spec in the package's vocabulary
# ---------------------------------------------------------------------------
def _displaced(lmk, amplitude, rng, modes=4):
    """lmk plus a smooth random displacement (low-frequency waves) whose largest component is ``amplitude``."""
    D = lmk.shape[0]
    disp = np.zeros_like(lmk)
    for _ in range(modes):
        k = rng.normal(size=D)
        k *= rng.uniform(1.0, 3.0) / np.linalg.norm(k)
        disp += rng.normal(size=(D, 1)) * np.cos(k @ lmk + rng.uniform(0.0, 2.0 * np.pi))[None, :]
    return lmk + disp * (amplitude / np.abs(disp).max())


@functools.lru_cache(maxsize=8)
def _strip(ang, lyr):
    obj = mesh.generate_element_object_2d(ang, lyr, [1, lyr])
    return obj, mesh.strip_nodes(ang, lyr)


@functools.lru_cache(maxsize=24)
def _annulus(ang, lyr):
    obj = api.build_element_object_2d(ang, lyr, [1, lyr], periodic=True)
    return obj, mesh.annulus_nodes(ang, lyr, 0.6, 1.0)


@functools.lru_cache(maxsize=12)
def _shell(level, lyr):
    surf, _, _, _, _, obj = mesh.shell_element_object(level, lyr, native=True)
    return obj, mesh.shell_nodes(surf, lyr, 0.7, 1.0)


def _with_target(spec, rng, amplitude, vfd):
    obj = spec["elmObj"]
    spec["tgt"] = mesh.varifold_target(_displaced(spec["lmkIniMat"], amplitude, rng), obj["vfdVtxMat"])
    spec["vfd"] = vfd
    return spec


def _frame_spec(c, rng):
    D = 2 if c["kind"] == "frame2d" else 3
    if D == 2:
        obj, lmk = _strip(c["ang"], c["lyr"])
        tau = np.array([rng.uniform(-1.5, 1.5), rng.uniform(-0.3, 0.5), 0.2, rng.uniform(0.3, 0.5)])
        prm, mod, width = np.array([1.0]), 3.0 * np.array([1.0, 1.0, 5.0]) * rng.uniform(0.9, 1.1), 0.2
    else:
        obj, lmk = _shell(c["level"], c["lyr"])
        cen = rng.normal(size=3)
        tau = np.concatenate([cen / np.linalg.norm(cen), [rng.uniform(0.4, 0.6)]])
        prm, mod, width = np.array([0.6, 1.0]), np.array([1.0, 1.0, 1.0, 5.0]) * rng.uniform(0.9, 1.1), 0.3
    spec = dict(dim=D, elaType="frame", lmkIniMat=_displaced(lmk, 0.01, rng), elmObj=obj, tauVarVec=tau,
                tauPrmVec=prm, modVec=mod, spdTanVal=0.625, spdTsvVal=0.125,
                ynkActPrmVec=np.array([0.01, 1.0, 4.0, 0.5]), reaActPrmVec=np.array([0.01, 1.0, 4.0, 0.5, 0.3]),
                ldmWgt=1e-2, knlOrder=c["order"], knlWidth=width, knlEps=1e-10, btmWgt=0.0, timeStp=0.01,
                timeNum=c["steps"] + 1, cgItrMax=10000, cgTolSqu=1e-24)
    return _with_target(spec, rng, 0.04, ("G", 0.5 if D == 2 else 0.3, "B", 1.0))


def _layered_spec(c, rng):
    two = "ang" in c
    obj, lmk = _annulus(c["ang"], c["lyr"]) if two else _shell(c["level"], c["lyr"])
    D, prisms = (2, c["lyr"] - 1) if two else (3, c["lyr"] - 1)
    L = min(c.get("materials", 3), prisms)
    of_prism = np.minimum((L * np.arange(prisms)) // prisms, L - 1)
    lyr = mesh.element_layers(obj["elmVtxMat"].shape[1], obj["elmPerLayer"], of_prism)
    lam = (2.0 if two else 3.0) ** np.arange(L) * rng.uniform(0.9, 1.1)
    col = []
    for _ in range(c.get("columns", 1)):
        cen = rng.normal(size=D)
        col.append(np.concatenate([cen / np.linalg.norm(cen), [rng.uniform(0.8, 1.0), rng.uniform(0.1, 0.2)]]))
    spec = dict(dim=D, elaType="isotropic", lmkIniMat=_displaced(lmk, 0.01, rng), elmObj=obj, elmLyrVec=lyr,
                tauVarVec=col[0], tauVarMat=np.array(col), tauPrmVec=np.zeros(2),
                modVec=np.column_stack([lam, lam / 2]).reshape(-1), spdLyrVec=0.01 * lam,
                ynkActPrmVec=np.array([0.5]), reaActPrmVec=np.array([2.0]), ldmWgt=0.0, knlOrder=1, knlWidth=0.1,
                knlEps=0.0, btmWgt=10.0, timeStp=0.02 if two else 0.01, timeNum=c["steps"] + 1, cgItrMax=20000,
                cgTolSqu=c["tol"] ** 2, rdItrMax=20000, rdTolSqu=c["tol"] ** 2)
    return _with_target(spec, rng, 0.04, ("G", 0.1, "B", 1.0) if two else ("M", 0.08, "B", 1.0))


def _varifold_spec(c, rng):
    if c["kind"] == "varifold2d":
        obj, lmk = _annulus(c["ang"], c["lyr"])
    else:
        obj, lmk = _shell(c["level"], c["lyr"])
    spec = dict(dim=lmk.shape[0], elmObj=obj, lmkIniMat=_displaced(lmk, 0.02, rng))
    return _with_target(spec, rng, 0.04, (c["cen"], c["width"], c["dir"], 0.8))


def _serve_specs(c, rng):
    sizes = np.random.default_rng(7)                       # the requests' sizes: the same for every seed
    out = []
    for k in range(c["requests"]):
        if k % 2 == 0:
            lyr = int(sizes.integers(6, 20))
            sub = dict(kind="layered2d", ang=int(sizes.integers(4, 14)) * lyr, lyr=lyr, materials=2 + k % 4)
        else:
            sub = dict(kind="layered3d", level=3 + k % 4 // 3, lyr=int(sizes.integers(4, 8)))
        out.append(_layered_spec(dict(sub, steps=c["steps"], tol=c["tol"]), rng))
    return out


def _inputs(c, seed):
    rng = np.random.default_rng(seed)
    if c["kind"].startswith("frame"):
        return _frame_spec(c, rng)
    if c["kind"].startswith("varifold"):
        return _varifold_spec(c, rng)
    if c["kind"] == "serve":
        return _serve_specs(c, rng)
    return _layered_spec(c, rng)


def prepare(case, seed):
    state = dict(case=case, spec=_inputs(case, seed))
    if case["kind"] == "serve":
        state["server"] = api.Server(hbm_budget=32e9, max_instances=64)   # the service a caller keeps running
    else:
        api.context()
    return state


# ---------------------------------------------------------------------------
# one call
# ---------------------------------------------------------------------------
def run(state):
    c, spec = state["case"], state["spec"]
    kind = c["kind"]
    if kind.startswith("frame"):
        r = api.forward(spec)
        return dict(lmk=r["lmkStk"], tau=r["tauMat"], obj=r["obj"])
    if kind.startswith("layered"):
        r = api.forward(spec, spec["tauVarMat"], precision=c["precision"], objective=c["objective"])
        out = dict(lmk=r["lmkStk"], tau=r["tauMat"])
        return dict(out, obj=r["obj"]) if c["objective"] else out
    if kind.startswith("varifold"):
        r = api.varifold(spec, spec["lmkIniMat"], grad=c["grad"], precision=c["precision"])
        return dict(obj=np.float64(r[0]), grad=r[1]) if c["grad"] else dict(obj=np.float64(r))
    if kind.startswith("adjoint"):
        r = api.adjoint(spec)
        return dict({k: r[k] for k in ("grad", "grad_layer", "grad_tau0", "grad_x0")}, obj=np.float64(r["obj"]))
    server = state["server"]
    ids = [server.submit(s, precision=c["precision"]) for s in spec]
    res = [server.result(i) for i in ids]
    return [dict(lmk=r["lmk"], tau=r["tau"], obj=np.float64(r["obj"])) for r in res]


# ---------------------------------------------------------------------------
# the work of one call
# ---------------------------------------------------------------------------
def _sizes(c):
    """(dim, nodes, elements, slots of the operator's pattern, boundary elements), from the mesh's structure."""
    if "ang" in c:
        around = c["ang"] - (1 if c["kind"].startswith("frame") else 0)      # segments of one node layer
        N, cells = c["ang"] * c["lyr"], around * (c["lyr"] - 1)
        edges = around * c["lyr"] + c["ang"] * (c["lyr"] - 1) + cells
        return 2, N, 2 * cells, N + 2 * edges, 2 * around
    V, F = 10 * 4 ** c["level"] + 2, 20 * 4 ** c["level"]
    N, p = V * c["lyr"], c["lyr"] - 1
    edges = (3 * F // 2) * (c["lyr"] + p) + V * p
    return 3, N, 3 * F * p, N + 2 * edges, F


def _pairs(dim, vd, vt, grad):
    """Flops of the varifold pair sums: the symmetric halves of both self terms and the cross term, each pair's
    squared distance, angle, two kernels and accumulation (an exponential counted as 20), the gradient's terms."""
    per = 3 * dim + 2 * dim + 30
    return (vd * vd / 2 + vt * vt / 2 + vd * vt) * per + ((vd * vd + vd * vt) * 8 * dim if grad else 0)


def _solve_work(c, steps, cols, objective, frame):
    """Per step: geometry and assembly of both operators, and one application of each per solve, the least any
    solver of the step needs; the frame model also evaluates its N x N kernel matrix and multiplies by it once."""
    D, N, E, Z, B = _sizes(c)
    flops = cols * steps * (E * (D + 1) ** 2 * (4 * D * D + 3 * D) + 2 * Z * (D * D + 1) + 40 * N * D)
    by = 4.0 * (E * (D + 1) + 2 * N * (D + 1) * E / N + 2 * Z + 4 * Z) + 8.0 * N * D
    by += 8.0 * N * (D + 1) * (steps + 1)
    if frame:
        flops += cols * steps * N * N * (2 * D + 30)
    if objective:
        flops += cols * _pairs(D, B, B, False)
    return by, flops


def work(case):
    c = case
    if c["kind"].startswith("varifold"):
        D, N, _, _, B = _sizes(c)
        return {"bytes": 8.0 * N * D * (2 if c["grad"] else 1) + 4.0 * B * D + 8.0 * B * (2 * D + 1),
                "flops": float(_pairs(D, B, B, c["grad"]))}
    if c["kind"] == "serve":
        by = fl = 0.0
        sizes = np.random.default_rng(7)
        for k in range(c["requests"]):
            if k % 2 == 0:
                lyr = int(sizes.integers(6, 20))
                sub = dict(kind="layered2d", ang=int(sizes.integers(4, 14)) * lyr, lyr=lyr)
            else:
                sub = dict(kind="layered3d", level=3 + k % 4 // 3, lyr=int(sizes.integers(4, 8)))
            b, f = _solve_work(sub, c["steps"], 1, True, False)
            by, fl = by + b, fl + f
        return {"bytes": by, "flops": fl}
    frame, adj = c["kind"].startswith("frame"), c["kind"].startswith("adjoint")
    by, fl = _solve_work(c, c["steps"], c.get("columns", 1), c.get("objective", True), frame)
    return {"bytes": by, "flops": fl * (3 if adj else 1)}


# ---------------------------------------------------------------------------
# the same results in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    a = np.ascontiguousarray(a)
    return torch.as_tensor(a, device=_dev()) if a.dtype == np.int64 else torch.as_tensor(
        a.astype(np.float64) if a.dtype.kind == "f" else a.astype(np.int64), device=_dev())


def _cg(A, b, prec, x, tol=1e-13, most=20000):
    """Conjugate gradients for the sparse A from x, to the relative residual tol, or until the residual has not
    fallen for 200 iterations."""
    shape, dot = b.shape, torch.dot
    b, x = b.reshape(-1), x.reshape(-1).clone()
    r = b - A @ x
    z = prec(r)
    p = z.clone()
    g = dot(r, z)
    goal = tol * float(b.norm())
    if goal == 0.0:
        return torch.zeros(shape, dtype=b.dtype, device=b.device)
    best, since = math.inf, 0
    for k in range(most):
        q = A @ p
        a = g / dot(p, q)
        x += a * p
        r -= a * q
        if k % 10 == 9:
            now = float(r.norm())
            since = 0 if now < 0.9 * best else since + 10
            best = min(best, now)
            if now <= goal or since >= 200:
                break
        z = prec(r)
        gn = dot(r, z)
        p = z + (gn / g) * p
        g = gn
    return x.reshape(shape)


class _Linear(torch.autograd.Function):
    """b -> A^-1 b for a symmetric A that is held constant."""

    @staticmethod
    def forward(ctx, b, solve):
        ctx.solve = solve
        return solve(b)

    @staticmethod
    def backward(ctx, g):
        return ctx.solve(g), None


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


class _Exact:
    """One forward solve; every operation differentiable when leaf tensors ask for gradients."""

    def __init__(self, spec):
        s = self.s = spec
        self.D = s["dim"]
        o = s["elmObj"]
        self.frame = s.get("elaType") == "frame"
        self.elm = _t(o["elmVtxMat"].T)                                    # E x (D+1)
        self.btm = _t(o["btmVtxMat"].T)
        self.N = s["lmkIniMat"].shape[1]
        pair = (self.elm[:, :, None] * self.N + self.elm[:, None, :]).reshape(-1)
        self.pattern, self.slot = torch.unique(pair, return_inverse=True)    # node pairs (row-major), E V V -> slot
        if self.frame:
            self.frm = _t((o["tanVtxMat"] if self.D == 2 else o["nmlVtxMat"]).T)
            self.tsv = _t(o["tsvVtxMat"].T)
        else:
            self.lyr = _t(s["elmLyrVec"].reshape(-1))
            mod = _t(np.asarray(s["modVec"]).reshape(-1, 2))
            self.lam, self.mu = mod[:, 0].clone(), mod[:, 1].clone()
            self.dif = _t(np.asarray(s["spdLyrVec"]))

    def scatter(self, idx, val):
        """Sum of val (E x k [x d]) at nodes idx (E x k)."""
        out = torch.zeros((self.N,) + val.shape[2:], dtype=torch.float64, device=val.device)
        return out.index_add(0, idx.reshape(-1), val.reshape((-1,) + val.shape[2:]))

    # geometry of a configuration: barycentric gradients, |det|, volume, frame
    def geometry(self, x):
        X = x[self.elm]
        q = X[:, 1:] - X[:, :1]
        if self.D == 2:
            det = q[:, 0, 0] * q[:, 1, 1] - q[:, 0, 1] * q[:, 1, 0]
            rot = lambda v: torch.stack([v[:, 1], -v[:, 0]], 1)
            g = torch.stack([rot(q[:, 1]), -rot(q[:, 0])], 1) / det[:, None, None]
        else:
            c = torch.stack([_cross(q[:, 1], q[:, 2]), _cross(q[:, 2], q[:, 0]), _cross(q[:, 0], q[:, 1])], 1)
            det = (q[:, 0] * c[:, 0]).sum(-1)
            g = c / det[:, None, None]
        g = torch.cat([-g.sum(1, keepdim=True), g], 1)
        ad = det.abs()
        geo = dict(x=x, g=g, ad=ad, vol=ad / math.factorial(self.D))
        if self.frame:
            F, S = x[self.frm], x[self.tsv]
            if self.D == 2:
                geo["f"] = _unit(_unit(F[:, 1] - F[:, 0]) + _unit(F[:, 3] - F[:, 2]))
                geo["s"] = _unit(_unit(S[:, 1] - S[:, 0]) + _unit(S[:, 3] - S[:, 2]))
            else:
                nml = lambda a: _unit(_cross(a[:, 1] - a[:, 0], a[:, 2] - a[:, 0]))
                geo["f"] = _unit(nml(F[:, :3]) + nml(F[:, 3:]))
                geo["s"] = _unit(sum(_unit(S[:, 2 * k + 1] - S[:, 2 * k]) for k in range(3)))
        else:
            geo["l"], geo["m"], geo["d"] = self.lam[self.lyr], self.mu[self.lyr], self.dif[self.lyr]
        w = float(self.s["btmWgt"])
        geo["pen"] = None
        if w != 0.0:
            B = x[self.btm]
            if self.D == 2:
                size = (B[:, 1] - B[:, 0]).norm(dim=-1)
            else:
                c = _cross(B[:, 1] - B[:, 0], B[:, 2] - B[:, 0])
                size = 0.5 * (c[:, 2].abs() if self.frame else c.norm(dim=-1))
            geo["pen"] = w * self.scatter(self.btm, (size / self.D)[:, None].expand(-1, self.D))
        return geo

    def stress(self, geo, F):
        """Stress of the velocity gradient F (E x D x D)."""
        I = torch.eye(self.D, dtype=torch.float64, device=F.device)
        tr = lambda a: a.diagonal(dim1=1, dim2=2).sum(-1)[:, None, None]
        if not self.frame:
            return geo["l"][:, None, None] * tr(F) * I + geo["m"][:, None, None] * (F + F.transpose(1, 2))
        e = 0.5 * (F + F.transpose(1, 2))
        f, s, mod = geo["f"], geo["s"], [float(v) for v in self.s["modVec"]]
        out = lambda a, b: a[:, :, None] * b[:, None, :]
        sym = lambda a, b: out(a, b) + out(b, a)
        es = (e @ s[:, :, None])[:, :, 0]
        ef = (e @ f[:, :, None])[:, :, 0]
        dot = lambda a, b: (a * b).sum(-1)[:, None, None]
        if self.D == 2:
            mT, mS, mA = mod[:3]
            return mT * dot(f, ef) * out(f, f) + mS * dot(s, es) * out(s, s) + mA * dot(f, es) * sym(f, s)
        lT, mT, mS, mA = mod[:4]
        return (lT * (tr(e) - dot(f, ef)) * (I - out(f, f)) + mT * (e - sym(ef, f) + dot(f, ef) * out(f, f))
                + mS * dot(s, es) * out(s, s) + mA * (sym(es, s) - dot(f, es) * sym(f, s)))

    def elastic(self, geo, v):
        F = v[self.elm].transpose(1, 2) @ geo["g"]
        f = (geo["vol"][:, None, None] * geo["g"]) @ self.stress(geo, F).transpose(1, 2)
        out = self.scatter(self.elm, f)
        return out if geo["pen"] is None else out + geo["pen"][:, None] * v

    def element_matrices(self, geo):
        """(E, V, D, V, D): the stiffness of every element."""
        E, D, g = self.elm.shape[0], self.D, geo["g"]
        out = torch.empty((E, D + 1, D, D + 1, D), dtype=torch.float64, device=g.device)
        for b in range(D + 1):
            for c in range(D):
                F = torch.zeros((E, D, D), dtype=torch.float64, device=g.device)
                F[:, c] = g[:, b]
                out[:, :, :, b, c] = (geo["vol"][:, None, None] * g) @ self.stress(geo, F).transpose(1, 2)
        return out

    def sparse(self, val):
        """CSR matrix from element matrices (E, V, k, V, k), and its k x k diagonal blocks."""
        N, k = self.N, val.shape[2]
        val = val.transpose(2, 3).reshape(-1, k, k)
        blk = torch.zeros((self.pattern.numel(), k, k), dtype=torch.float64, device=val.device)
        blk.index_add_(0, self.slot, val)
        row, col = self.pattern // N, self.pattern % N
        diag = blk[row == col]
        d = torch.arange(k, device=val.device)
        count = torch.bincount(row, minlength=N)
        start = torch.cumsum(count, 0) - count
        # entry (r, c) of block s of row i sits in matrix row i k + r, at place (s - start_i) k + c of that row
        place = (start[row] * k * k)[:, None, None] + d[None, :, None] * (count[row] * k)[:, None, None] \
            + ((torch.arange(row.numel(), device=val.device) - start[row]) * k)[:, None, None] + d[None, None, :]
        cols, vals = torch.empty(blk.numel(), dtype=torch.int64, device=val.device), torch.empty_like(blk.reshape(-1))
        cols[place.reshape(-1)] = (col[:, None, None] * k + d[None, None, :]).expand(-1, k, k).reshape(-1)
        vals[place.reshape(-1)] = blk.reshape(-1)
        crow = torch.cat([torch.zeros(1, dtype=torch.int64, device=val.device),
                          torch.cumsum(torch.repeat_interleave(count * k, k), 0)])
        return torch.sparse_csr_tensor(crow, cols, vals, (N * k, N * k)), diag

    def solve_spd(self, A, prec, apply, b, guess, diff):
        """A^-1 b; with diff, A's and b's derivatives are carried by one more step through apply (A as a function)."""
        with torch.no_grad():
            v = _cg(A, b.detach(), prec, guess.detach())
        if not diff:
            return v
        return v + _Linear.apply(b - apply(v), lambda r: _cg(A, r.detach(), prec, torch.zeros_like(r)))

    def velocity(self, geo, b, K, guess, diff):
        with torch.no_grad():
            if K is not None:
                return self.velocity_frame(geo, b, K)
            me = self.element_matrices(geo)
            A, blocks = self.sparse(me)
            if geo["pen"] is not None:
                blocks = blocks + geo["pen"][:, None, None] * torch.eye(self.D, dtype=b.dtype, device=b.device)
                A = A + torch.sparse_csr_tensor(torch.arange(self.N * self.D + 1, device=b.device),
                                                torch.arange(self.N * self.D, device=b.device),
                                                geo["pen"].repeat_interleave(self.D), tuple(A.shape))
            inv = torch.linalg.inv(blocks)
            prec = lambda r: (inv @ r.reshape(self.N, self.D, 1)).reshape(-1)
        return self.solve_spd(A, prec, lambda v: self.elastic(geo, v), b, guess, diff)

    def velocity_frame(self, geo, b, K):
        """(ldm K^-1 + E) v = b as (ldm I + E K) w = b, v = K w, by a dense factorisation."""
        N, D = self.N, self.D
        A = self.sparse(self.element_matrices(geo))[0].to_dense().reshape(N * D, N, D)
        if geo["pen"] is not None:
            i = torch.arange(N, device=b.device)
            for d in range(D):
                A[i * D + d, i, d] += geo["pen"]
        B = torch.empty((N * D, N, D), dtype=torch.float64, device=b.device)
        for d in range(D):
            B[:, :, d] = A[:, :, d] @ K
        B = B.reshape(N * D, N * D)
        B.diagonal().add_(float(self.s["ldmWgt"]))
        return K @ torch.linalg.solve(B, b.reshape(-1)).reshape(N, D)

    def kernel(self, x):
        """RKHS matrix: Matern of the given order (Gaussian for -1) plus eps on the diagonal."""
        s, w = self.s, float(self.s["knlWidth"])
        d2 = sum((x[:, None, d] - x[None, :, d]) ** 2 for d in range(self.D))
        o = s["knlOrder"]
        if o == -1:
            K = torch.exp(-d2 / (w * w))
        elif self.D == 3:
            r = d2.sqrt() / w
            c = {0: [1], 1: [1, 1], 2: [1, 1, 1 / 3], 3: [1, 1, 2 / 5, 1 / 15], 4: [1, 1, 3 / 7, 2 / 21, 1 / 105]}[o]
            K = sum(a * r ** k for k, a in enumerate(c)) * torch.exp(-r)
        else:
            r = d2.sqrt() / w
            q = r * r
            near = r < 2.3e-16
            rr = torch.where(near, torch.ones_like(r), r)
            f0 = torch.where(near | (r > 700), torch.zeros_like(r), q * torch.special.modified_bessel_k0(rr))
            f1 = torch.where(near, torch.ones_like(r), torch.where(r > 700, torch.zeros_like(r),
                                                                   rr * torch.special.modified_bessel_k1(rr)))
            K = {0: lambda: f1, 1: lambda: f0 / 2 + f1, 2: lambda: f0 / 2 + (1 + q / 8) * f1,
                 3: lambda: (0.5 + q / 48) * f0 + (1 + q / 6) * f1,
                 4: lambda: (0.5 + q / 32) * f0 + (1 + 3 * q / 16 + q * q / 384) * f1}[o]()
        K.diagonal().add_(float(s["knlEps"]))
        return K

    def activity(self, tau):
        y, r = [float(v) for v in self.s["ynkActPrmVec"]], [float(v) for v in self.s["reaActPrmVec"]]
        if not self.frame:
            return y[0] * tau, r[0] * tau * (1.0 - tau)
        return y[2] * _yank(2.0 * (tau - y[0]) / (y[1] - y[0]) - 1.0, y[3]), \
            r[2] * _reaction(2.0 * (tau - r[0]) / (r[1] - r[0]) - 1.0, r[3], r[4])

    def mass(self, geo, u):
        """M u: consistent mass, |det| / 24 (2D) or / 120 (3D) times (1 + delta_ab)."""
        U = u[self.elm]
        return self.scatter(self.elm, (geo["ad"] / (24.0 if self.D == 2 else 120.0))[:, None]
                            * (U + U.sum(1, keepdim=True)))

    def flux(self, geo, grad):
        if not self.frame:
            return geo["d"][:, None] * grad
        a, b = float(self.s["spdTanVal"]), float(self.s["spdTsvVal"])
        along = lambda v: (grad * v).sum(-1, keepdim=True) * v
        return (a * along(geo["f"]) if self.D == 2 else a * (grad - along(geo["f"]))) + b * along(geo["s"])

    def diffusion(self, geo, u):
        flux = self.flux(geo, (u[self.elm][:, None, :] @ geo["g"])[:, 0])
        return self.scatter(self.elm, (geo["vol"][:, None, None] * geo["g"] @ flux[:, :, None])[:, :, 0])

    def reaction_matrices(self, geo, dt):
        """(E, V, 1, V, 1): mass plus dt diffusion of every element."""
        g, V = geo["g"], self.D + 1
        fl = torch.stack([self.flux(geo, g[:, b]) for b in range(V)], 2)                  # E x D x V
        unit = (torch.ones((V, V), dtype=g.dtype, device=g.device) + torch.eye(V, dtype=g.dtype, device=g.device))
        m = (geo["ad"] / (24.0 if self.D == 2 else 120.0))[:, None, None] * unit
        return (m + dt * geo["vol"][:, None, None] * (g @ fl))[:, :, None, :, None]

    def start(self, x, p):
        d2 = lambda c: ((x - c) ** 2).sum(-1)
        D, tp = self.D, [float(v) for v in np.atleast_1d(self.s["tauPrmVec"])]
        if not self.frame:
            return p[D] * torch.exp(-d2(p[:D]) / (2.0 * p[D + 1] ** 2))
        c, h, rad, power = (p[:2], p[2], p[3], int(tp[0])) if D == 2 else (p[:3], p[3], tp[0], int(tp[1]))
        q = d2(c) / (rad * rad)
        return torch.where(q < 1.0, h * (1.0 - (1.0 - (q - 1.0) ** 2) ** power), torch.zeros_like(q))

    def solve(self, x, p, diff=False, dtau0=None):
        """Trajectory: lists of positions (N x D) and concentrations, timeNum long."""
        dt, D = float(self.s["timeStp"]), self.D
        useK = self.frame or float(self.s["ldmWgt"]) != 0.0
        tau = self.start(x, p)
        if dtau0 is not None:
            tau = tau + dtau0
        xs, ts, geo, v = [x], [tau], self.geometry(x), torch.zeros_like(x)
        for _ in range(int(self.s["timeNum"]) - 1):
            fy, fr = self.activity(tau)
            mean = fy[self.elm].mean(1)
            b = self.scatter(self.elm, -(mean * geo["vol"])[:, None, None] * geo["g"])
            v = self.velocity(geo, b, self.kernel(x) if useK else None, v, diff)
            x = x + dt * v
            nxt = self.geometry(x)
            rhs = self.mass(geo, tau + dt * fr)
            with torch.no_grad():
                A, diag = self.sparse(self.reaction_matrices(nxt, dt))
                diag = diag.reshape(-1)
            tau = self.solve_spd(A, lambda r, d=diag: r / d,
                                 lambda u, at=nxt: self.mass(at, u) + dt * self.diffusion(at, u), rhs, tau, diff)
            geo = nxt
            xs.append(x)
            ts.append(tau)
        return xs, ts

    def objective(self, x):
        return _varifold(self.s, x)


def _yank(t, w):
    a = 3 * (w - 2) / (w ** 3 * (6 + w * (w - 6)))
    b = (6 + w * (8 * w - 15)) / (3 * (w - 2))
    c = 6 / (6 + w * (w - 6))
    up, down = a * (1 + t) ** 3 * (t - b), a * (1 - t) ** 3 * (-t - b)
    y = torch.where(t < -1 + w, up, torch.where(t < 1 - w, 1 - c * t * t, down))
    return torch.where((t < -1) | (t >= 1), torch.zeros_like(t), y)


def _reaction(t, w, a):
    h = 24 * (a - 1) + a * w * (w - 12)
    k = 6 * (a - 1) + a * w * (w - 6)
    b1 = 8 * k / (3 * w ** 4)
    b2 = -(144 * (a - 1) + w * (24 * (5 - 11 * a) + w * (156 * a - 29 * a * w))) / (24 * k)
    c1 = -h / (9 * w ** 3)
    c2 = -(24 * (a - 1) + w * (12 * (2 - 3 * a) + a * w * (13 + 2 * w))) / (3 * w ** 3)
    c3 = -((w - 1) ** 2) * h / (3 * w ** 3)
    c4 = -(24 * (a - 1) + w * (12 * (6 - 7 * a) + w * (109 * a - 72 + w * (3 * (5 - 21 * a) + a * w * (15 - w))))) \
        / (9 * w ** 3)
    half = lambda u: torch.where(u < -1 + 0.5 * w, b1 * (1 + u) ** 3 * (u - b2), c4 + u * (c3 + u * (c2 + u * c1)))
    y = torch.where(t < -1 + w, half(t), torch.where(t < 1 - w, 1 - a * t * t, half(-t)))
    return torch.where((t < -1) | (t >= 1), torch.zeros_like(t), y)


def _elements(x, vtx):
    """Centres, unit directions and sizes of the boundary elements vtx (n x D) of nodes x (N x D)."""
    X = x[vtx]
    if x.shape[1] == 2:
        d = X[:, 1] - X[:, 0]
        return X.mean(1), _unit(d), d.norm(dim=-1)
    c = _cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0])
    return X.mean(1), _unit(c), 0.5 * c.norm(dim=-1)


def _pair_sum(A, B, vfd):
    """Sum over all pairs of k_centre k_direction size size, in row chunks recomputed for the gradient."""
    ck, cw, dk, dw = vfd

    def rows(ca, ua, va, cb, ub, vb):
        d2 = sum((ca[:, None, d] - cb[None, :, d]) ** 2 for d in range(ca.shape[1])) / (cw * cw)
        if ck == "G":
            k = torch.exp(-d2)
        elif ck == "C":
            k = 1.0 / (1.0 + d2)
        else:
            zero = d2 == 0.0
            r = torch.where(zero, torch.ones_like(d2), d2).sqrt()
            k = torch.where(zero, torch.ones_like(d2), (1.0 + r) * torch.exp(-r))
        t = ua @ ub.T
        if dk == "B":
            k = k * t * t
        elif dk == "L":
            k = k * t
        else:
            k = k * torch.exp(2.0 * ((t if dk == "O" else t * t) - 1.0) / (dw * dw))
        return va @ (k @ vb)

    total, step = 0.0, max(1, (1 << 25) // max(1, B[0].shape[0]))
    for i in range(0, A[0].shape[0], step):
        part = [a[i:i + step] for a in A] + list(B)
        if any(p.requires_grad for p in part):
            total = total + torch.utils.checkpoint.checkpoint(rows, *part, use_reentrant=False)
        else:
            total = total + rows(*part)
    return total


def _varifold(spec, x):
    D = _elements(x, _t(spec["elmObj"]["vfdVtxMat"].T))
    cen, uni, vol = spec["tgt"]
    T = (_t(np.asarray(cen).T), _t(np.asarray(uni).T), _t(vol))
    return _pair_sum(D, D, spec["vfd"]) - 2.0 * _pair_sum(D, T, spec["vfd"]) + _pair_sum(T, T, spec["vfd"])


def _forward(spec, columns, objective):
    e, objs = _Exact(spec), []
    x0 = _t(spec["lmkIniMat"].T)
    with torch.no_grad():
        for col in columns:
            xs, ts = e.solve(x0, _t(col))
            if objective:
                objs.append(float(e.objective(xs[-1])))
    return torch.stack(xs).transpose(1, 2), torch.stack(ts), np.array(objs)


def exact(case, seed):
    c, spec = case, _inputs(case, seed)
    kind = c["kind"]
    if kind.startswith("frame"):
        lmk, tau, obj = _forward(spec, [spec["tauVarVec"]], True)
        return dict(lmk=lmk.cpu().numpy(), tau=tau.cpu().numpy(), obj=obj)
    if kind.startswith("layered"):
        lmk, tau, obj = _forward(spec, spec["tauVarMat"], c["objective"])
        out = dict(lmk=lmk.cpu().numpy(), tau=tau.cpu().numpy())
        return dict(out, obj=obj) if c["objective"] else out
    if kind.startswith("varifold"):
        x = _t(spec["lmkIniMat"].T).requires_grad_(c["grad"])
        obj = _varifold(spec, x)
        if not c["grad"]:
            return dict(obj=np.float64(obj.item()))
        (g,) = torch.autograd.grad(obj, x)
        return dict(obj=np.float64(obj.detach().item()), grad=g.T.contiguous().cpu().numpy())
    if kind.startswith("adjoint"):
        e = _Exact(spec)
        x, p = _t(spec["lmkIniMat"].T).requires_grad_(), _t(spec["tauVarVec"]).requires_grad_()
        d0 = torch.zeros(e.N, dtype=torch.float64, device=_dev(), requires_grad=True)
        leaves = [x, p, d0] + [t.requires_grad_() for t in (e.lam, e.mu, e.dif)]
        xs, _ = e.solve(x, p, True, d0)
        obj = e.objective(xs[-1])
        gx, gp, g0, gl, gm, gd = torch.autograd.grad(obj, leaves, materialize_grads=True)
        return dict(obj=np.float64(obj.detach().item()), grad=gp.cpu().numpy(),
                    grad_layer=torch.stack([gl, gm, gd], 1).contiguous().cpu().numpy(), grad_tau0=g0.cpu().numpy(),
                    grad_x0=gx.T.contiguous().cpu().numpy())
    out = []
    for s in spec:
        lmk, tau, obj = _forward(s, [s["tauVarVec"]], True)
        out.append(dict(lmk=lmk[-1].contiguous().cpu().numpy(), tau=tau[-1].cpu().numpy(), obj=obj[0]))
    return out
