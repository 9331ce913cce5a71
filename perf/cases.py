"""Measured cases: what users of this framework run, through its Python entry points.

The framework does one thing, the quasi-static Newton step of a solid-mechanics problem, and is
called in six ways:

  solve     StaticMatrix.solve: a whole load-stepped Newton solve of one mesh (FP64 or mixed);
  batch     BatchedStaticMatrix.solve: many uneven tetrahedral problems in one context;
  adjoint   autograd.equilibrium_displacement: a forward solve and its backward pass;
  linear    ConjugateGradient.solve: the linear-solver plugin on a caller's CSR matrix;
  assemble  update_internal_variables + assemble: the element-level drop-in, host K and f_int;
  apply     update_internal_variables + the matrix-free tangent products.

Sizes, materials and boundary conditions are those of neon_b200.problem's configurations and of
the tests (20^3 linear elasticity, neo-Hooke up to 64^3, J2 up to 100^3, the microsphere models
with a shear-modulus field, batches of 8^3 to 40^3 tetrahedral cubes); solves that take many
increments there take one or two here.  J2 solves stay below yield: past it neon's update, which
mutates the plastic strain on every Newton iteration, makes the solution depend on the last bits of
every iterate, so no two correct solvers agree; plastic points are measured by `assemble`.

`exact` restates the same mechanics in plain torch FP64 and solves it to round-off.
"""
import math

import numpy as np
import torch

from neon_b200 import api, autograd
from neon_b200 import mesh as mesh_module
from neon_b200 import problem as P

# ------------------------------------------------------------------------------------------
# cases
# ------------------------------------------------------------------------------------------


def listed():
    return [
        # the smallest whole call: the 27-element cube of neon's own examples, two increments
        {"name": "solve_neohooke_3", "kind": "solve", "element": "hex8", "model": "neohooke",
         "bc": "rollers", "nx": 3, "ny": 3, "nz": 3, "steps": 2, "precision": "fp64"},
        # the 20^3 linear-elastic configuration: an everyday mesh, where launches and latency count
        {"name": "solve_linear_20", "kind": "solve", "element": "hex8", "model": "linear",
         "bc": "clamped", "nx": 20, "ny": 20, "nz": 20, "steps": 1, "precision": "fp64"},
        # a middle-sized ragged block of rubber
        {"name": "solve_neohooke_37x29x32", "kind": "solve", "element": "hex8",
         "model": "neohooke", "bc": "rollers", "nx": 37, "ny": 29, "nz": 32, "steps": 1,
         "precision": "fp64"},
        # the neo-Hooke configuration at its own size, first increment, mixed precision
        {"name": "solve_neohooke_64_mixed", "kind": "solve", "element": "hex8",
         "model": "neohooke", "bc": "rollers", "nx": 64, "ny": 64, "nz": 64, "steps": 1,
         "precision": "mixed"},
        # the J2 configuration at its own size (3M DOFs), first increment, both precisions
        {"name": "solve_j2_100", "kind": "solve", "element": "hex8", "model": "j2",
         "bc": "clamped", "nx": 100, "ny": 100, "nz": 100, "steps": 1, "precision": "fp64"},
        {"name": "solve_j2_100_mixed", "kind": "solve", "element": "hex8", "model": "j2",
         "bc": "clamped", "nx": 100, "ny": 100, "nz": 100, "steps": 1, "precision": "mixed"},
        # the Langevin microsphere under traction with a modulus field (anisotropic tangent)
        {"name": "solve_langevin_20", "kind": "solve", "element": "hex8", "model": "langevin",
         "bc": "traction", "nx": 20, "ny": 20, "nz": 20, "steps": 1, "precision": "fp64"},
        # parameter identification: forward solve and gradient of a modulus field
        {"name": "adjoint_microsphere_24", "kind": "adjoint", "element": "hex8",
         "model": "microsphere", "bc": "traction", "nx": 24, "ny": 24, "nz": 24, "steps": 1,
         "precision": "fp64"},
        # batched uneven tetrahedral problems, both precisions
        {"name": "batch_neohooke_8_16", "kind": "batch", "element": "tet4", "model": "neohooke",
         "bc": "rollers", "instances": 24, "lo": 8, "hi": 16, "sizes": 11, "steps": 1,
         "precision": "fp64"},
        {"name": "batch_neohooke_12_28_mixed", "kind": "batch", "element": "tet4",
         "model": "neohooke", "bc": "rollers", "instances": 16, "lo": 12, "hi": 28, "sizes": 12,
         "steps": 1, "precision": "mixed"},
        # the linear-solver plugin on a caller's matrix
        {"name": "linear_24", "kind": "linear", "element": "hex8", "model": "linear",
         "bc": "clamped", "nx": 24, "ny": 24, "nz": 24},
        # the element-level drop-in with plastic points
        {"name": "assemble_j2_40", "kind": "assemble", "element": "hex8", "model": "j2",
         "bc": "clamped", "nx": 40, "ny": 40, "nz": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "batch", "adjoint", "linear",
                       "assemble", "apply"])
    if kind == "batch":
        lo = rng.randint(4, 12)
        return {"kind": "batch", "element": "tet4", "model": "neohooke", "bc": "rollers",
                "instances": _log_int(rng, 3, 24), "lo": lo, "hi": lo + rng.randint(2, 12),
                "sizes": rng.randint(1, 10 ** 6), "steps": 1,
                "precision": rng.choice(["fp64", "mixed"])}
    cap = {"solve": 60, "adjoint": 24, "linear": 30, "assemble": 40, "apply": 60}[kind]
    n = _log_int(rng, 4, cap)
    dims = [max(2, int(round(n * rng.uniform(0.6, 1.0)))) for _ in range(3)]
    case = {"kind": kind, "element": "hex8", "nx": dims[0], "ny": dims[1], "nz": dims[2]}
    if kind == "adjoint":
        return dict(case, model=rng.choice(["microsphere", "langevin"]), bc="traction", steps=1,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "linear":
        return dict(case, model="linear", bc="clamped")
    if kind == "assemble":
        return dict(case, element=rng.choice(["hex8", "hex8", "tet4"]),
                    model=rng.choice(["j2", "neohooke", "linear", "microsphere", "langevin"]),
                    bc="clamped")
    if kind == "apply":
        return dict(case, element=rng.choice(["hex8", "hex8", "tet4"]),
                    model=rng.choice(["j2", "neohooke", "linear"]), bc="clamped")
    model = rng.choice(["linear", "neohooke", "neohooke", "j2", "microsphere", "langevin"])
    bc = {"linear": "clamped", "j2": "clamped", "neohooke": "rollers"}.get(model, "traction")
    if model == "langevin":
        case.update({k: min(case[k], 32) for k in ("nx", "ny", "nz")})
    if model in ("linear", "neohooke") and rng.random() < 0.3:
        case.update({k: min(case[k], 30) for k in ("nx", "ny", "nz")}, element="tet4")
    return dict(case, model=model, bc=bc, steps=rng.choice([1, 1, 2]),
                precision=rng.choice(["fp64", "fp64", "mixed"]))


# ------------------------------------------------------------------------------------------
# inputs: mesh, material, boundary conditions of one seed
# ------------------------------------------------------------------------------------------
_TETS = ((0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6), (0, 5, 1, 6))


def _box(element, dims, jitter, rng):
    """Nodes, connectivity and integer lattice coordinates of a box of nx x ny x nz cells whose
    longest side is 1; interior nodes are moved by up to `jitter` cells."""
    nx, ny, nz = dims
    top = max(dims)
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    ijk = np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1)
    X = ijk / float(top)
    inner = np.all((ijk > 0) & (ijk < np.array(dims)), axis=1)
    X[inner] += rng.uniform(-jitter, jitter, size=(int(inner.sum()), 3)) / top
    K, J, I = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    I, J, K = I.ravel(), J.ravel(), K.ravel()
    c = [(I + a) + (nx + 1) * ((J + b) + (ny + 1) * (K + d)) for a, b, d in
         ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))]
    conn = np.stack(c, axis=1)
    if element == "tet4":
        conn = conn[:, np.array(_TETS)].reshape(-1, 4)
        e = [X[conn[:, a]] - X[conn[:, 3]] for a in range(3)]
        flip = np.einsum("ij,ij->i", e[0], np.cross(e[1], e[2])) < 0
        conn[flip, 0], conn[flip, 1] = conn[flip, 1].copy(), conn[flip, 0].copy()
    return X, conn.astype(np.int32), ijk


def _material(model, scale):
    if model in ("linear", "j2"):
        E, nu = 200e3 * scale, 0.3
        K, G = E / (3 * (1 - 2 * nu)), E / (2 * (1 + nu))
        if model == "linear":
            return P.Material(P.LINEAR_ELASTIC, K, G)
        return P.Material(P.J2_SMALL_STRAIN, K, G, 200.0, 1e3)
    if model == "neohooke":
        return P.Material(P.NEO_HOOKE, 10.0 * scale, scale)
    kind = P.GAUSS_AFFINE_MICROSPHERE if model == "microsphere" else P.LANGEVIN_AFFINE_MICROSPHERE
    return P.Material(kind, 100.0, 1.0, segments_per_chain=50.0)


def _inputs(case, seed):
    """Everything a problem is made of, as plain arrays (shared by prepare and exact)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    dims = (case["nx"], case["ny"], case["nz"])
    model = case["model"]
    X, conn, ijk = _box(case["element"], dims, 0.05 if model == "j2" else 0.1, rng)
    scale = float(rng.uniform(0.8, 1.25))
    mat = _material(model, scale if model in ("linear", "neohooke") else 1.0)
    load = float(rng.uniform(0.8, 1.2))
    Ge = None
    if model in ("microsphere", "langevin"):
        Ge = rng.lognormal(0.0, 0.3, size=conn.shape[0]) * mat.G
    height = dims[2] / max(dims)
    steps = case.get("steps", 1)
    side = [np.flatnonzero(ijk[:, d] == 0) for d in range(3)]
    top = np.flatnonzero(ijk[:, 2] == dims[2])
    fixed, amount = [], []  # (dofs, final value)
    force = None
    if case["bc"] == "rollers":
        fixed = [3 * side[d] + d for d in range(3)] + [3 * top + 2]
        amount = [0.0, 0.0, 0.0, 0.03 * load * steps * height]
    else:
        fixed = [3 * side[2] + d for d in range(3)]
        amount = [0.0, 0.0, 0.0]
        if case["bc"] == "clamped":
            fixed.append(3 * top + 2)
            amount.append({"linear": 1e-3, "j2": 3e-4}.get(model, 1e-3) * load * height)
        else:  # consistent nodal forces of a uniform traction on the (regular) top face
            w = np.zeros(X.shape[0])
            tx, ty = ijk[top, 0], ijk[top, 1]
            share = (np.where((tx > 0) & (tx < dims[0]), 2, 1) *
                     np.where((ty > 0) & (ty < dims[1]), 2, 1))
            w[top] = share * 0.25 / max(dims) ** 2
            force = (3 * top + 2, w[top], 0.05 * load)
    return {"X": X, "conn": conn, "ijk": ijk, "mat": mat, "model": model, "Ge": Ge,
            "fixed": fixed, "amount": amount, "force": force, "steps": steps, "rng": rng}


def _problem(d, name):
    tol = {"linear": 1e-6, "microsphere": 1e-9, "langevin": 1e-9}.get(d["model"], 1e-8)
    dt = 1.0 / d["steps"]
    opts = P.Options(residual_tolerance=tol, displacement_tolerance=tol, linear_iterations=15,
                     period=1.0, initial=dt, minimum=dt, maximum=dt, adaptive=False,
                     cg_tolerance=1e-10, cg_maximum_iterations=200000)
    times = np.array([0.0, 1.0])
    tables = [P.DofTable(dofs.astype(np.int32), times, np.array([0.0, a]))
              for dofs, a in zip(d["fixed"], d["amount"])]
    forces = []
    if d["force"] is not None:
        dofs, w, value = d["force"]
        forces = [P.DofTable(dofs.astype(np.int32), times, np.array([0.0, value]), weights=w)]
    return P.Problem(name, mesh_module.Mesh(d["X"], d["conn"], {}), d["mat"], tables, opts,
                     nodal_forces=forces, element_shear_modulus=d["Ge"])


def _batch_sizes(case):
    rng = np.random.Generator(np.random.PCG64(case["sizes"]))
    return [int(v) for v in rng.integers(case["lo"], case["hi"] + 1, size=case["instances"])]


def _batch_inputs(case, seed):
    out = []
    for i, m in enumerate(_batch_sizes(case)):
        d = _inputs(dict(case, nx=m, ny=m, nz=m), seed * 1009 + i)
        d["mat"] = P.Material(P.NEO_HOOKE, 20.0 * d["mat"].G, d["mat"].G)
        d["amount"][-1] *= 2.0 / 3.0
        out.append(d)
    return out


def _field(d, kind):
    """A displacement a program would hand to the element drop-ins: the load's stretch plus
    nodal noise; for J2 well past yield in part of the block."""
    size = d["X"].max(axis=0)
    u = np.zeros_like(d["X"])
    u[:, 2] = {"j2": 1.5e-3, "linear": 1e-3}.get(d["model"], 0.1) * d["X"][:, 2] ** 2 / size[2]
    h = 1.0 / max(d["ijk"].max(axis=0))
    noise = {"j2": 2e-4, "linear": 1e-3}.get(d["model"], 0.02)
    u += d["rng"].uniform(-noise, noise, size=u.shape) * h
    return u.ravel()


def prepare(case, seed):
    kind = case["kind"]
    precision = api.MIXED if case.get("precision") == "mixed" else api.FP64
    if kind == "batch":
        problems = [_problem(d, "instance %d" % i)
                    for i, d in enumerate(_batch_inputs(case, seed))]
        return {"kind": kind, "batch": api.BatchedStaticMatrix(problems, precision=precision)}
    d = _inputs(case, seed)
    if kind == "solve":
        return {"kind": kind,
                "static_matrix": api.StaticMatrix(_problem(d, "solve"), precision=precision)}
    if kind == "adjoint":
        g = np.zeros(3 * d["X"].shape[0])
        g[2::3] = d["rng"].uniform(0.0, 1.0, size=d["X"].shape[0]) / d["X"].shape[0]
        return {"kind": kind, "problem": _problem(d, "adjoint"), "precision": precision,
                "G": torch.from_numpy(d["Ge"]), "weights": torch.from_numpy(g)}
    if kind == "linear":
        rp, ci, v, b = _linear_system(d)
        return {"kind": kind, "A": (rp, ci, v), "b": b, "x": np.zeros_like(b),
                "solver": api.ConjugateGradient(1e-12, 100000)}
    mesh = api.SolidMesh(d["X"], d["conn"], d["mat"], d["Ge"])
    state = {"kind": kind, "mesh": mesh, "u": _field(d, kind)}
    if kind == "apply":
        state["v"] = d["rng"].standard_normal(state["u"].size)
    return state


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return state["static_matrix"].solve()
    if kind == "batch":
        return state["batch"].solve()
    if kind == "adjoint":
        G = state["G"].clone().requires_grad_(True)
        u = autograd.equilibrium_displacement(G, state["problem"], state["precision"])
        (u * state["weights"]).sum().backward()
        return {"u": u.detach(), "gradient": G.grad}
    if kind == "linear":
        return state["solver"].solve(state["A"], state["x"], state["b"])
    mesh = state["mesh"]
    mesh.save_internal_variables(False)  # from the last committed plastic state
    mesh.update_internal_variables(state["u"])
    if kind == "assemble":
        K, f = mesh.assemble()
        return {"K": K, "f": f}
    # the FP32 product is handed back in FP64; it has FP32 accuracy
    return {"y": mesh.apply_tangent(state["v"]),
            "y32": torch.from_numpy(mesh.apply_tangent_fp32(state["v"])).float()}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _counts(case):
    if case["kind"] == "batch":
        cells = [m ** 3 for m in _batch_sizes(case)]
        nodes = [(m + 1) ** 3 for m in _batch_sizes(case)]
        longest = _batch_sizes(case)
    else:
        dims = (case["nx"], case["ny"], case["nz"])
        cells = [dims[0] * dims[1] * dims[2]]
        nodes = [(dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1)]
        longest = [max(dims)]
    tet = case["element"] == "tet4"
    return [(6 * c if tet else c, n, m) for c, n, m in zip(cells, nodes, longest)]


def work(case):
    """Bytes: inputs once and results once; an iterative solve also reads and writes its iterate,
    residual and direction once per CG iteration.  Operations: the element integrals once per
    Newton iteration and one product with the tangent per CG iteration.  Iteration counts of the
    Jacobi-CG grow with the number of cells along the longest side; the factors are typical."""
    tet = case["element"] == "tet4"
    npe, row = (4, 15) if tet else (8, 27)
    bytes_, flops = 0.0, 0.0
    for E, N, m in _counts(case):
        mesh = 4.0 * npe * E + 24.0 * N
        integrals = (1552.0 if tet else 32240.0) * E
        product = 2.0 * 9.0 * row * N
        kind = case["kind"]
        if kind in ("assemble", "apply"):
            state = 112.0 * 8 * E if case["model"] == "j2" and not tet else 0.0
            bytes_ += mesh + 48.0 * N + state + (8.0 * 9 * row * N if kind == "assemble" else 0)
            flops += integrals + (0.0 if kind == "assemble" else 2 * product)
            continue
        per = 8.0 if case["model"] in ("linear", "j2") else 20.0
        newton = 1 if kind == "linear" else 4 * case.get("steps", 1)
        cg = per * m * newton
        bytes_ += newton * mesh + cg * 6 * 24.0 * N
        flops += newton * integrals + cg * product
        if kind == "linear":
            bytes_ += 12.0 * 9 * row * N
        if kind == "adjoint":
            bytes_ += 2 * per * m * 6 * 24.0 * N
            flops += 2 * per * m * product
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------------------------------
# the same mechanics in plain torch, FP64
# ------------------------------------------------------------------------------------------
_W1, _W2, _W3 = 2 * 0.0265214244093, 2 * 0.0199301476312, 2 * 0.0250712367487
_D0, _D1, _D2 = 0.707106781187, 0.387907304067, 0.836095596749


def _sphere(dev):
    """The 21-point unit-sphere rule of Bazant and Oh (1986), half the sphere."""
    r = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
    for a, b in ((0, 1), (0, 2), (1, 2)):
        for s in (1, -1):
            v = [0.0, 0.0, 0.0]
            v[a], v[b] = _D0, s * _D0
            r.append(tuple(v))
    for big in (2, 1, 0):
        for s in (1, -1):
            for t in (1, -1):
                v = [_D1, s * _D1, t * _D1]
                v[big] *= _D2 / _D1
                r.append(tuple(v))
    w = [_W1] * 3 + [_W2] * 6 + [_W3] * 12
    return (torch.tensor(r, dtype=torch.float64, device=dev),
            torch.tensor(w, dtype=torch.float64, device=dev))


def _shape(element, dev):
    """Reference gradients [points, nodes, 3] and weights."""
    if element == "tet4":
        dN = torch.tensor([[[1., 0, 0], [0, 1, 0], [0, 0, 1], [-1, -1, -1]]], dtype=torch.float64)
        return dN.to(dev), torch.tensor([1.0 / 6.0], dtype=torch.float64, device=dev)
    c = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1],
                      [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=torch.float64)
    q = c / math.sqrt(3.0)
    f = 1.0 + c[None] * q[:, None]  # [point, node, axis]
    dN = torch.stack([c[None, :, 0] * f[..., 1] * f[..., 2], c[None, :, 1] * f[..., 0] * f[..., 2],
                      c[None, :, 2] * f[..., 0] * f[..., 1]], dim=-1) / 8.0
    return dN.to(dev), torch.ones(8, dtype=torch.float64, device=dev)


def _det_inv(A):
    a, b, c = A[..., 0, :], A[..., 1, :], A[..., 2, :]
    bc, ca, ab = (torch.linalg.cross(p, q, dim=-1) for p, q in ((b, c), (c, a), (a, b)))
    det = (a * bc).sum(-1)
    return det, torch.stack([bc, ca, ab], dim=-1) / det[..., None, None]


class _Body:
    def __init__(self, X, conn, model, K, G, mat, element, Ge=None):
        self.dev = dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.X = torch.as_tensor(X, dtype=torch.float64, device=dev)
        self.conn = torch.as_tensor(np.asarray(conn, np.int64), device=dev)
        self.model, self.mat = model, mat
        per = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev).reshape(-1, 1)  # noqa: E731
        self.K, self.G = per(K), per(G if Ge is None else Ge)
        self.dN, self.w = _shape(element, dev)
        if model in ("microsphere", "langevin"):
            self.sphere = _sphere(dev)
        self.F0 = torch.einsum("eai,qak->eqik", self.X[self.conn], self.dN)
        _, self.F0i = _det_inv(self.F0)
        self.N = self.X.shape[0]
        self.I = torch.eye(3, dtype=torch.float64, device=dev)

    def stress(self, H, G):
        """Cauchy stress and the tangent's lam', mu', and for J2 b and N."""
        I, model = self.I, self.model
        K, G = self.K[..., None, None], G[..., None, None]
        lam = K - 2 * G / 3
        extra = None
        if model in ("linear", "j2"):
            eps = 0.5 * (H + H.mT)
            s = lam * torch.diagonal(eps, dim1=-2, dim2=-1).sum(-1)[..., None, None] * I + 2 * G * eps
            lt, mt = lam.expand_as(s[..., :1, :1]), G.expand_as(s[..., :1, :1])
            if model == "j2":
                dev = s - torch.diagonal(s, dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3 * I
                dn = torch.sqrt((dev * dev).sum((-1, -2)))[..., None, None]
                vm = math.sqrt(1.5) * dn
                f = vm - self.mat.yield_stress
                on = f > 0
                h3 = 3 * G + self.mat.hardening
                dg = torch.where(on, f / h3, torch.zeros_like(f))
                n = dev / torch.where(dn > 0, dn, torch.ones_like(dn))
                s = s - 2 * G * dg * math.sqrt(1.5) * n
                c1 = torch.where(on, dg * 6 * G * G / vm, torch.zeros_like(dg))
                c2 = torch.where(on, 6 * G * G * (dg / vm - 1 / h3), torch.zeros_like(dg))
                lt, mt = lam + c1 / 3, G - c1 / 2
                extra = (c2, n)
            return s, lt, mt, extra
        F = I + H
        J, _ = _det_inv(F)
        J = J[..., None, None]
        if model == "neohooke":
            B = F @ F.mT
            return (lam * torch.log(J) * I + G * (B - I)) / J, lam, G - lam * torch.log(J), None
        r, w = self.sphere
        t = torch.einsum("eqij,sj->eqsi", J ** (-1.0 / 3.0) * F, r)
        l2 = (t * t).sum(-1)
        Nc = self.mat.segments_per_chain
        chain = 3.0 * torch.ones_like(l2) if model == "microsphere" else (3 * Nc - l2) / (Nc - l2)
        tau = G * torch.einsum("eqs,eqsi,eqsj->eqij", w * chain, t, t)
        p = J * K / 2 * (J - 1 / J)
        trt = torch.diagonal(tau, dim1=-2, dim2=-1).sum(-1)[..., None, None]
        s = (p * I + tau - trt / 3 * I) / J
        if model == "langevin":
            ps = (l2 * l2 + 3 * Nc * Nc) / (Nc - l2) ** 2
            m = torch.einsum("eqsi,eqsj->eqsij", t, t) - l2[..., None, None] / 3 * I
            extra = (G[..., None] * (w * (ps - chain) / l2)[..., None, None], m)
        kappa = J * J * (K / 2 * (1 + 1 / (J * J)))
        return s, kappa + p - 2.0 / 9.0 * trt, trt / 3 - p, extra

    def points(self, u, G):
        u = u.reshape(-1, 3)
        U = torch.einsum("eai,qak->eqik", u[self.conn], self.dN)
        det, Ji = _det_inv(self.F0 + U)
        L = torch.einsum("qak,eqkj->eqaj", self.dN, Ji)
        return L, self.w * det, self.stress(U @ self.F0i, G)

    def scatter(self, y):
        out = torch.zeros(self.N, 3, dtype=torch.float64, device=self.dev)
        return out.index_add(0, self.conn.reshape(-1), y.reshape(-1, 3)).reshape(-1)

    def force(self, u, G=None):
        L, s, (sig, _, _, _) = self.points(u, self.G if G is None else G)
        return self.scatter(torch.einsum("eq,eqij,eqaj->eai", s, sig, L))

    def blocks(self, u):
        """The element stiffness of the framework's tangent, [E, a, i, b, k]."""
        L, s, (sig, lt, mt, extra) = self.points(u, self.G)
        Q = s.shape
        full = lambda v: v[..., 0, 0].expand(Q) * s  # noqa: E731
        LL = torch.einsum("eqai,eqbi->eqab", L, L)
        Ke = torch.einsum("eq,eqai,eqbk->eaibk", full(lt), L, L)
        Ke += torch.einsum("eq,eqak,eqbi->eaibk", full(mt), L, L)
        diag = torch.einsum("eq,eqab->eab", full(mt), LL)
        if self.model not in ("linear", "j2"):
            diag += torch.einsum("eq,eqai,eqij,eqbj->eab", s, L, sig, L)
        Ke += torch.einsum("eab,ik->eaibk", diag, self.I)
        if self.model == "j2":
            NL = torch.einsum("eqij,eqaj->eqai", extra[1], L)
            Ke += torch.einsum("eq,eqai,eqbk->eaibk", full(extra[0]), NL, NL)
        elif self.model == "langevin":
            c = extra[0][..., 0, 0] * s[..., None]
            for d in range(c.shape[-1]):
                mL = torch.einsum("eqij,eqaj->eqai", extra[1][:, :, d], L)
                Ke += torch.einsum("eq,eqai,eqbk->eaibk", c[..., d], mL, mL)
        return Ke

    def csr(self, Ke):
        """Sorted CSR of the assembled matrix, explicit zeros kept."""
        dofs = (3 * self.conn[:, :, None] + torch.arange(3, device=self.dev)).reshape(
            self.conn.shape[0], -1)
        m = dofs.shape[1]
        rows, cols = dofs[:, :, None].expand(-1, m, m), dofs[:, None, :].expand(-1, m, m)
        n = 3 * self.N
        key, where = torch.unique((rows * n + cols).reshape(-1), return_inverse=True)
        val = torch.zeros(key.numel(), dtype=torch.float64, device=self.dev).index_add(
            0, where, Ke.reshape(-1))
        r = torch.div(key, n, rounding_mode="floor")
        rp = torch.zeros(n + 1, dtype=torch.int64, device=self.dev)
        rp[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
        return rp, key - r * n, val

    def product(self, Ke, v):
        y = torch.einsum("eaibk,ebk->eai", Ke, v.reshape(-1, 3)[self.conn])
        return self.scatter(y)

    def diagonal(self, Ke):
        return self.scatter(torch.einsum("eaiai->eai", Ke))


def _cg(product, inv, b, tol, most=20000):
    x = torch.zeros_like(b)
    r, z = b.clone(), inv * b
    p, rz, stop = z.clone(), (b * z).sum(), tol * tol * float((b * b).sum())
    if stop == 0.0:
        return x
    for it in range(most):
        q = product(p)
        a = rz / (p * q).sum()
        x, r = x + a * p, r - a * q
        if it % 8 == 7 and float((r * r).sum()) <= stop:
            break
        z = inv * r
        new = (r * z).sum()
        p, rz = z + (new / rz) * p, new
    return x


def _body(d, element):
    return _Body(d["X"], d["conn"], d["model"], d["mat"].K, d["mat"].G, d["mat"], element, d["Ge"])


def _equilibrium(body, fixed, amount, force, steps):
    """u with f_int(u) = f_ext on the free DOFs, and the mask of the free DOFs."""
    n, dev = 3 * body.N, body.dev
    free = torch.ones(n, dtype=torch.float64, device=dev)
    final = torch.zeros(n, dtype=torch.float64, device=dev)
    for dofs, a in zip(fixed, amount):
        at = torch.as_tensor(np.asarray(dofs, np.int64), device=dev)
        free[at], final[at] = 0.0, torch.as_tensor(a, dtype=torch.float64, device=dev)
    fext = torch.zeros(n, dtype=torch.float64, device=dev)
    for dofs, w, value in force:
        fext[torch.as_tensor(np.asarray(dofs, np.int64), device=dev)] += value * torch.as_tensor(
            w, dtype=torch.float64, device=dev)
    u = torch.zeros(n, dtype=torch.float64, device=dev)
    for step in range(1, steps + 1):
        prescribed = (1 - free) * (final * step / steps - u)
        for it in range(40):
            Ke = body.blocks(u)
            r = fext * step / steps - body.force(u)
            if it == 0:
                r = r - body.product(Ke, prescribed)
                u = u + prescribed
            r = r * free
            d = body.diagonal(Ke)
            du = _cg(lambda p: free * body.product(Ke, p), 1.0 / d, r, 1e-9)
            u = u + du
            if float(du.norm()) <= 1e-14 * float(u.norm()):
                break
            if it > 3 and float(du.norm()) <= 3e-13 * float(u.norm()):
                break
    return u, free


def _linear_system(d):
    """CSR arrays of a clamped linear-elastic stiffness and a load vector (host)."""
    body = _body(d, "hex8")
    rp, ci, v = body.csr(body.blocks(torch.zeros(3 * body.N, dtype=torch.float64,
                                                 device=body.dev)))
    fixed = torch.zeros(3 * body.N, dtype=torch.bool, device=body.dev)
    for dofs in d["fixed"]:
        fixed[torch.as_tensor(np.asarray(dofs, np.int64), device=body.dev)] = True
    rows = torch.repeat_interleave(torch.arange(3 * body.N, device=body.dev), rp[1:] - rp[:-1])
    v[(fixed[rows] | fixed[ci]) & (rows != ci)] = 0.0
    b = torch.from_numpy(d["rng"].standard_normal(3 * body.N)).to(body.dev)
    b[fixed] = 0.0
    return (rp.to(torch.int32).cpu().numpy(), ci.to(torch.int32).cpu().numpy(), v.cpu().numpy(),
            b.cpu().numpy())


def _exact_adjoint(body, u, free, g):
    """-lambda^T df_int/dG with (df_int/du)^T lambda = g on the free DOFs."""
    K = body.blocks(u)
    inv = 1.0 / body.diagonal(K)
    ug = u.clone().requires_grad_(True)
    f = body.force(ug)

    def transposed(v):
        return free * torch.autograd.grad(f, ug, v, retain_graph=True)[0]

    lam = torch.zeros_like(g)
    for _ in range(40):
        r = free * g - transposed(lam)
        d = _cg(lambda p: free * body.product(K, p), inv, r, 1e-7)
        lam = lam + d
        if float(d.norm()) <= 1e-14 * float(lam.norm()):
            break
    Gg = body.G.clone().requires_grad_(True)
    return -torch.autograd.grad((lam * body.force(u, Gg)).sum(), Gg)[0].reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    size = sum(E * m for E, _, m in _counts(case))
    if kind in ("solve", "adjoint") and size > 1.6e6 or kind == "batch" and size > 5e6:
        return None
    if kind in ("assemble", "apply") and (size > 3e6 or case["model"] == "langevin" and size > 4e5):
        return None
    if kind == "batch":
        ds = _batch_inputs(case, seed)
        off = np.cumsum([0] + [d["X"].shape[0] for d in ds])
        E = [d["conn"].shape[0] for d in ds]
        body = _Body(np.concatenate([d["X"] for d in ds]),
                     np.concatenate([d["conn"] + o for d, o in zip(ds, off)]), "neohooke",
                     np.repeat([d["mat"].K for d in ds], E), np.repeat([d["mat"].G for d in ds], E),
                     None, "tet4")
        fixed = [x + 3 * o for d, o in zip(ds, off) for x in d["fixed"]]
        amount = [a for d in ds for a in d["amount"]]
        return _equilibrium(body, fixed, amount, [], case["steps"])[0].cpu().numpy()
    d = _inputs(case, seed)
    if kind == "linear":
        rp, ci, v, b = (torch.from_numpy(a) for a in _linear_system(d))
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        A = torch.sparse_csr_tensor(rp.long(), ci.long(), v, size=(len(b), len(b))).to(dev)
        rows = torch.repeat_interleave(torch.arange(len(b)), (rp[1:] - rp[:-1]).long())
        inv = torch.empty_like(b)
        inv[rows[rows == ci]] = 1.0 / v[rows == ci]
        inv, b = inv.to(dev), b.to(dev)
        x = torch.zeros_like(b)
        for _ in range(4):  # residuals replaced: to round-off
            x = x + _cg(lambda p: A @ p, inv, b - A @ x, 1e-8)
        return x.cpu().numpy()
    body = _body(d, case["element"])
    if kind in ("solve", "adjoint"):
        u, free = _equilibrium(body, d["fixed"], d["amount"],
                               [] if d["force"] is None else [d["force"]], case["steps"])
        if kind == "solve":
            return u.cpu().numpy()
        g = np.zeros(3 * body.N)
        g[2::3] = d["rng"].uniform(0.0, 1.0, size=body.N) / body.N
        grad = _exact_adjoint(body, u, free, torch.from_numpy(g).to(body.dev))
        return {"u": u.cpu().numpy(), "gradient": grad.cpu().numpy()}
    u = torch.from_numpy(_field(d, kind)).to(body.dev)
    Ke = body.blocks(u)
    if kind == "assemble":
        return {"K": body.csr(Ke)[2].cpu().numpy(), "f": body.force(u).cpu().numpy()}
    v = torch.from_numpy(d["rng"].standard_normal(3 * body.N)).to(body.dev)
    y = body.product(Ke, v).cpu().numpy()
    return {"y": y, "y32": y}
