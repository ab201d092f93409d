"""The work that users of this framework have it do, as cases that can be timed and checked.

Every case goes through the package's public entry points (`FemModel`,
`ElasticModel`, `density_objectives`) on the meshes of `mesh.py`: the lognormal
and density cantilevers and the J2 bar, at their own sizes, at the smallest ones
where launches and latency count, and at odd ones.

kinds
  linear    one static solve K x = b by Jacobi-PCG (FP64, or FP32 iterations
            with FP64 refinement), matrix resident
  multigrid the same solve with the geometric multigrid preconditioner
  block     several load cases solved together
  design    one step of a density optimisation: objectives and gradients at the
            current design, objectives at a trial design, each reassembled
  newton    one Newton-Raphson increment of the J2 bar past first yield
  assemble  reassembly of the stiffness and the products K x with it
  post      loads, internal force, stresses and reactions of a given displacement
  analysis  the whole linear analysis, from the mesh in host memory to stresses
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__ as _entry

ufc = _entry.load_package()
from ufc_fem_kernel_b200 import adjoint  # noqa: E402  (importable once the package is loaded)

DEVICE = 0
E0 = 210e3


# --------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest solve: a handful of elements, bound by launches and latency
        {"name": "linear_10x2x2_fp64", "kind": "linear", "nx": 10, "ny": 2, "nz": 2, "precision": "fp64",
         "storage": "full", "numbering": "box", "buffers": "cuda"},
        # the slender 40x8x8 cantilever, refined request on the symmetric storage (the matrix stays in L2)
        {"name": "linear_40x8x8_refine", "kind": "linear", "nx": 40, "ny": 8, "nz": 8, "precision": "refine",
         "storage": "symmetric", "numbering": "box", "buffers": "cuda"},
        # an ordinary mesh of odd sizes whose nodes are numbered without structure, buffers in host memory
        {"name": "linear_61x33x29_fp64_shuffled", "kind": "linear", "nx": 61, "ny": 33, "nz": 29, "precision": "fp64",
         "storage": "full", "numbering": "shuffled", "buffers": "host"},
        # the largest: 5.4M DOF, FP32 iterations with FP64 refinement on the symmetric storage
        {"name": "linear_192x96x96_refine", "kind": "linear", "nx": 192, "ny": 96, "nz": 96, "precision": "refine",
         "storage": "symmetric", "numbering": "box", "buffers": "cuda"},
        # 1.6M DOF with multigrid, the solver for a structured box
        {"name": "multigrid_128x64x64", "kind": "multigrid", "nx": 128, "ny": 64, "nz": 64, "cycle": "fp32",
         "storage": "symmetric"},
        # sixteen load cases in one block solve
        {"name": "block16_64x32x32", "kind": "block", "nx": 64, "ny": 32, "nz": 32, "nrhs": 16},
        # one step of a density optimisation with four load cases, forward and backward
        {"name": "design_64x32x32", "kind": "design", "nx": 64, "ny": 32, "nz": 32, "nrhs": 4, "solver": "multigrid"},
        # one plastic increment of the J2 bar at its own size
        {"name": "newton_64x32x32_jacobi", "kind": "newton", "nx": 64, "ny": 32, "nz": 32, "solver": "jacobi"},
        # a smaller bar with the multigrid inner solver: tangents and hierarchies rebuilt per iteration
        {"name": "newton_32x16x16_multigrid", "kind": "newton", "nx": 32, "ny": 16, "nz": 16, "solver": "multigrid"},
        # new moduli on a 1.6M-DOF mesh: assembly of every form the refined solver reads, then K x
        {"name": "assemble_128x64x64", "kind": "assemble", "nx": 128, "ny": 64, "nz": 64, "storage": "symmetric",
         "numbering": "box"},
        # everything either side of the solve on a mesh of odd sizes
        {"name": "post_97x51x47", "kind": "post", "nx": 97, "ny": 51, "nz": 47, "numbering": "box"},
        # a whole linear analysis from host arrays: model, pattern, loads, assembly, solve, stresses
        {"name": "analysis_48x24x24", "kind": "analysis", "nx": 48, "ny": 24, "nz": 24, "numbering": "box"},
    ]


# largest number of elements a drawn case of each kind may have
_CAP = {"linear": 400_000, "multigrid": 524_288, "block": 65_536, "design": 65_536, "newton": 40_000,
        "assemble": 524_288, "post": 524_288, "analysis": 65_536}


def draw(rng):
    kind = rng.choice(["linear", "linear", "multigrid", "block", "design", "newton", "assemble", "post", "analysis"])
    n = math.exp(rng.uniform(math.log(60.0), math.log(float(_CAP[kind]))))
    side = (n / 2.0) ** (1.0 / 3.0)  # about twice as long as wide and high
    dims = [max(1, int(round(f * side * rng.uniform(0.75, 1.25)))) for f in (2.0, 1.0, 1.0)]
    case = {"kind": kind}
    boxes = kind in ("multigrid", "design", "newton")  # boxes that halve at least twice
    if boxes:
        step = 4 if side < 12 else 8
        dims = [max(step, int(round(d / step)) * step) for d in dims]
    case.update(nx=max(2, dims[0]), ny=dims[1], nz=dims[2])
    while case["nx"] * case["ny"] * case["nz"] > _CAP[kind]:
        case["nx"] -= 8 if boxes else 1
    numbering = rng.choice(["box", "box", "shuffled"])
    storage = rng.choice(["full", "symmetric"])
    if kind == "linear":
        case.update(precision=rng.choice(["fp64", "refine"]), storage=storage, numbering=numbering,
                    buffers=rng.choice(["cuda", "cuda", "host"]))
    elif kind == "multigrid":
        case.update(cycle=rng.choice(["fp32", "fp64"]), storage=storage)
    elif kind == "block":
        case.update(nrhs=rng.choice([2, 3, 5, 8, 16, 16, 24, 32]))
        while case["nx"] * case["ny"] * case["nz"] * case["nrhs"] > 16 * 65_536:
            case["nrhs"] -= 8
    elif kind == "design":
        case.update(nrhs=rng.randint(1, 4), solver=rng.choice(["multigrid", "jacobi"]))
    elif kind == "newton":
        case.update(solver=rng.choice(["jacobi", "multigrid"]))
    elif kind == "assemble":
        case.update(storage=storage, numbering=numbering)
    else:
        case.update(numbering=numbering)
    return case


# --------------------------------------------------------------------------- inputs
def _rng(seed, salt):
    return np.random.default_rng([int(seed), salt])


def _distort(p, seed):
    """Interior nodes of the box moved by up to a tenth of the spacing: element shapes of an ordinary mesh."""
    nx, ny, nz = p.shape
    h = p.coords.max(axis=0) / np.array(p.shape)
    lo, hi = p.coords.min(axis=0), p.coords.max(axis=0)
    inner = np.all((p.coords > lo + 0.5 * h) & (p.coords < hi - 0.5 * h), axis=1)
    p.coords[inner] += _rng(seed, 1).uniform(-0.1, 0.1, size=(int(inner.sum()), 3)) * h


def _shuffle(p, seed):
    """The same problem with nodes and elements numbered at random."""
    r = _rng(seed, 2)
    node = r.permutation(p.n_nodes)  # new id of each node
    elem = r.permutation(p.n_elems)
    coords = np.empty_like(p.coords)
    coords[node] = p.coords
    p.coords = coords
    p.conn = np.ascontiguousarray(node[p.conn].astype(np.int32)[elem])
    p.props = np.ascontiguousarray(p.props[elem])
    dof = 3 * node[p.fixed // 3] + p.fixed % 3
    order = np.argsort(dof)
    p.fixed = dof[order].astype(np.int32)
    p.fixed_values = p.fixed_values[order]
    f = np.empty_like(p.f)
    f.reshape(-1, 3)[node] = p.f.reshape(-1, 3)
    p.f = f
    p.meta["node"] = node
    p.meta["elem_new"] = np.argsort(elem)  # new id of each old element


def _problem(case, seed):
    """The problem a case stands for, made from the seed alone."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kind = case["kind"]
    if kind in ("block", "design"):
        p = ufc.mesh.density_problem(nx, ny, nz, seed=seed, n_rhs=1)
        tip = np.nonzero(p.coords[:, 0] == nx)[0]
        F = np.zeros((case["nrhs"], p.n_dof))
        F[:, 3 * tip + 2] = -(1.0 + 0.5 * _rng(seed, 3).standard_normal((case["nrhs"], tip.size)))
        p.meta["F"] = F
        return p
    if kind == "newton":
        p = ufc.mesh.j2_bar(nx, ny, nz)
        p.props[:, 2] *= 1.0 + 0.05 * np.clip(_rng(seed, 4).standard_normal(p.n_elems), -3, 3)  # yield stress
        return p
    if (nx, ny, nz) == (40, 8, 8):  # the slender cantilever's own box
        p = ufc.mesh.cantilever(nx, ny, nz, 10.0, 2.0, 2.0, E=ufc.mesh.lognormal_moduli(nx * ny * nz, seed))
    else:
        p = ufc.mesh.lognormal_cantilever(nx, ny, nz, seed)
    if kind in ("assemble", "post", "analysis"):
        _distort(p, seed)
    if case.get("numbering") == "shuffled":
        _shuffle(p, seed)
    return p


def _build(case):
    b = ufc.BUILD_FP64
    if case.get("precision") == "refine" or case["kind"] in ("assemble", "analysis"):
        b |= ufc.BUILD_FP32_ROUNDED
    if case.get("storage") == "symmetric" or case["kind"] == "analysis":
        b |= ufc.BUILD_SYMMETRIC
    return b


def _algo(case):
    if case["kind"] == "multigrid" or case.get("solver") == "multigrid":
        return ufc.SolverAlgo(tolerance=1e-10, precond_type=ufc.SOLV_PREC_MG)
    if case.get("precision") == "refine" or case["kind"] == "analysis":
        return ufc.SolverAlgo(tolerance=1e-10, precision_mode=ufc.PRECISION_FP32_REFINE)
    return ufc.SolverAlgo(tolerance=1e-10)


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(torch.device("cuda", DEVICE))


def _loaded_faces(p, case, seed):
    """Faces of the x = max side (face 6, outward normal +x), a traction per face and a pressure per face."""
    nx, ny, nz = p.shape
    e = np.array([nx - 1 + nx * (j + ny * k) for k in range(nz) for j in range(ny)], dtype=np.int32)
    r = _rng(seed, 5)
    t = np.array([0.0, 0.0, -1.0]) + 0.2 * r.standard_normal((e.size, 3))
    q = 0.5 + 0.1 * r.standard_normal(e.size)
    if "elem_new" in p.meta:
        e = p.meta["elem_new"][e].astype(np.int32)
    return e, np.full(e.size, 6, dtype=np.int32), t, q


def _displacement(p, seed):
    """A bent and stretched bar with a little roughness, of the size a solve gives."""
    r = _rng(seed, 6)
    x, y, z = p.coords.T / p.coords.max()
    a = r.uniform(0.5, 1.5, size=6)
    u = np.stack([1e-3 * (a[0] * x * (z - 0.25) + 0.3 * a[1] * x * x), 1e-3 * a[2] * (0.2 * x * y - 0.1 * np.sin(3 * x)),
                  -1e-3 * (a[3] * x * x + 0.1 * a[4] * np.sin(2 * x + a[5]))], axis=1)
    u += 1e-6 * r.standard_normal(u.shape)
    u = u.ravel()
    u[p.fixed] = 0.0
    return u


def _direction(p, seed):
    """A search direction of an iterative solver: rough, zero on the fixed DOFs."""
    x = _rng(seed, 8).standard_normal(p.n_dof)
    x[p.fixed] = 0.0
    return x


def prepare(case, seed):
    kind = case["kind"]
    p = _problem(case, seed)
    s = {"case": case, "kind": kind, "algo": _algo(case)}
    if kind == "analysis":
        s["p"] = p
        s["faces"] = _loaded_faces(p, case, seed)
        return s
    if kind == "design":
        m = adjoint.ElasticModel(p, device=DEVICE)
        r = _rng(seed, 7)
        s["rho"] = _cuda(p.meta["rho"])
        s["trial"] = _cuda(np.clip(p.meta["rho"] + 0.02 * r.standard_normal(p.n_elems), 0.3, 1.0))
        s["F"] = _cuda(p.meta["F"]) * m.free
        s["tip"] = 3 * int(p.meta["tip_node"]) + 2
        m.set_moduli(E0 * s["trial"] ** 3)
        if case["solver"] == "multigrid":
            m.fem.mg_setup(*p.shape, precision=ufc.PRECISION_FP32_REFINE)
        s["model"] = m
        return s
    m = ufc.FemModel.from_problem(p, device=DEVICE)
    s["model"] = m
    if kind == "newton":
        # two elastic increments and one past first yield, committed; the next one is the case
        lin = ufc.SolverAlgo(tolerance=1e-10)
        if case["solver"] == "multigrid":
            m.internal_force(m.displacement(), update_state=True)
            m.assemble(ufc.BUILD_FP64)
            m.mg_setup(*p.shape)
        for step in _COMMITTED:
            m.nr_increment(_target(p, step), lin=s["algo"] if case["solver"] == "multigrid" else lin)
            m.commit()
        s["target"] = _cuda(_target(p, _INCREMENT))
        s["u"] = torch.empty(p.n_dof, dtype=torch.float64, device=torch.device("cuda", DEVICE))
        return s
    if kind == "post":
        s["u"] = _cuda(_displacement(p, seed))
        s["faces"] = [_cuda(a) for a in _loaded_faces(p, case, seed)]
        return s
    m.assemble(_build(case))
    if kind == "assemble":
        s["build"] = _build(case)
        s["x"] = _cuda(_direction(p, seed))
        s["x32"] = s["x"].float()
        return s
    if kind == "block":
        B = p.meta["F"].copy()
        B[:, p.fixed] = 0.0
        s["B"] = _cuda(B)
        return s
    b = ufc.lifted_rhs(m, p.f, p.fixed_values)
    s["b"] = b if case.get("buffers") == "host" else _cuda(b)
    if kind == "multigrid":
        m.mg_setup(*p.shape,
                   precision=ufc.PRECISION_FP32_REFINE if case["cycle"] == "fp32" else ufc.PRECISION_FP64)
    return s


_COMMITTED, _INCREMENT, _STEPS = (2, 4), 5, 20


def _target(p, step):
    return ufc.mesh.j2_bar_target(p, step, n_steps=_STEPS)


# --------------------------------------------------------------------------- one pass
def run(state):
    return _RUN[state["kind"]](state)


def _run_linear(s):
    x, _ = s["model"].solve(s["b"], s["algo"])
    return x


def _run_block(s):
    X, _ = s["model"].solve_block(s["B"], s["algo"])
    return X


def _run_design(s):
    m = s["model"]
    rho = s["rho"].clone().requires_grad_(True)
    F = s["F"].clone().requires_grad_(True)
    J1, J2, U = adjoint.density_objectives(rho, F, m, s["algo"], s["tip"])
    g_rho, g_F = torch.autograd.grad(J1 + J2, [rho, F])
    with torch.no_grad():  # line search: the objectives at a trial design
        T1, T2, V = adjoint.density_objectives(s["trial"], s["F"], m, s["algo"], s["tip"])
    return {"J1": J1.detach(), "J2": J2.detach(), "U": U.detach(), "g_rho": g_rho, "g_F": g_F, "trial_J1": T1,
            "trial_J2": T2, "trial_U": V}


def _run_newton(s):
    m = s["model"]
    m.rollback()
    m.nr_increment(s["target"], lin=s["algo"])
    return m.displacement(out=s["u"])


def _run_assemble(s):
    m = s["model"]
    m.assemble(s["build"])
    return m.spmv(s["x"]), m.spmv(s["x32"], precision=ufc.PRECISION_FP32_REFINE)


def _run_post(s):
    m, u = s["model"], s["u"]
    elem, face, traction, pressure = s["faces"]
    f = m.load_faces(elem, face, traction=traction, pressure=pressure)
    fint, r, rnorm, fnorm = m.internal_force(u, f_ext=f, update_state=False)
    sig, vm = m.stress(u)
    nodal, nodal_vm = m.stress_nodal(u)
    rf = m.reactions(u, f_ext=f)
    return {"f": f, "fint": fint, "r": r, "rnorm": rnorm, "fint_norm": fnorm, "sigma": sig, "von_mises": vm,
            "nodal": nodal, "nodal_von_mises": nodal_vm, "reactions": rf}


def _run_analysis(s):
    p = s["p"]
    elem, face, traction, pressure = s["faces"]
    m = ufc.FemModel.from_problem(p, device=DEVICE)
    m.assemble(_build(s["case"]))
    f = m.load_faces(elem, face, traction=traction, pressure=pressure)
    u, _ = m.solve(ufc.lifted_rhs(m, f, p.fixed_values), s["algo"])
    _, vm = m.stress(u, want_sigma=False)
    nodal, _ = m.stress_nodal(u)
    rf = m.reactions(u, f_ext=f)
    m.close()
    return {"u": u, "von_mises": vm, "nodal": nodal, "reactions": rf}


_RUN = {"linear": _run_linear, "multigrid": _run_linear, "block": _run_block, "design": _run_design,
        "newton": _run_newton, "assemble": _run_assemble, "post": _run_post, "analysis": _run_analysis}


# --------------------------------------------------------------------------- work
def work(case):
    """Bytes and flops a pass cannot do without.  A solve counts the iterations
    its method needs on these problems (measured: Jacobi-PCG about 16 nx in FP64
    and 22 nx refined, multigrid 15) times one read of the upper half of the
    block matrix and of the iteration's vectors; element work counts the
    symmetric Ke or B^T sigma of every element once."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kind = case["kind"]
    N, E = (nx + 1) * (ny + 1) * (nz + 1), nx * ny * nz
    n, G = 3 * N, 8 * E
    blocks = (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)  # coupled node pairs of a box
    upper = (blocks + N) // 2
    it64 = {"bytes": 72.0 * upper + 88.0 * n, "flops": 18.0 * blocks + 12.0 * n}
    it32 = {"bytes": 36.0 * upper + 52.0 * n, "flops": 18.0 * blocks + 12.0 * n}
    mesh = 24.0 * N + 32.0 * E + 16.0 * E
    ke = 36 * 8 * 22.0 * E  # 36 node pairs, 8 Gauss points
    fint = 8 * 600.0 * E
    asm = {"bytes": mesh + 72.0 * upper, "flops": ke}

    def times(w, k):
        return {q: k * v for q, v in w.items()}

    def plus(*ws):
        return {q: sum(w[q] for w in ws) for q in ("bytes", "flops")}

    mg_it = plus(it64, times(it32, 4 * 8.0 / 7.0))
    io = {"bytes": 16.0 * n, "flops": 0.0}
    if kind == "linear":
        return plus(io, times(it64, 16 * nx) if case["precision"] == "fp64" else times(it32, 22 * nx))
    if kind == "multigrid":
        return plus(io, times(mg_it, 15))
    if kind == "block":
        k, its = case["nrhs"], 16 * nx
        return {"bytes": its * (72.0 * upper + 88.0 * n * k), "flops": its * k * (18.0 * blocks + 12.0 * n)}
    if kind == "design":
        solve = times(mg_it, 15) if case["solver"] == "multigrid" else times(it64, 16 * nx)
        sens = {"bytes": case["nrhs"] * 16.0 * n + 8.0 * E, "flops": case["nrhs"] * 8 * 250.0 * E}
        return plus(times(asm, 2), times(solve, 3 * case["nrhs"]), sens)
    if kind == "newton":
        solve = times(mg_it, 30) if case["solver"] == "multigrid" else times(it64, 28 * nx)
        one = plus({"bytes": G * (13 * 16.0 + 288.0), "flops": G * 600.0 + fint},
                   {"bytes": 288.0 * G + 72.0 * upper, "flops": 36 * 8 * 162.0 * E}, solve)
        return times(one, 4)
    if kind == "assemble":
        sym = {"bytes": 36.0 * upper, "flops": 0.0}
        return plus(asm, sym, it64, it32)
    out = {"bytes": 8.0 * (7 * G + 7 * N + 4 * n), "flops": 3 * fint}
    post = plus({"bytes": 3 * mesh + 24.0 * n, "flops": 0.0}, out)
    if kind == "post":
        return post
    return plus({"bytes": mesh, "flops": 0.0}, asm, times(it32, 22 * nx), post)


# --------------------------------------------------------------------------- the values in 64 bits
# A restatement in torch, FP64: the 8-node hexahedron with the 2x2x2 rule,
# element matrices applied one by one, CG with a Jacobi preconditioner, the J2
# return map with linear hardening.
_SIGN = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                      [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=torch.float64)


def _gauss():
    g = 1.0 / math.sqrt(3.0)
    return torch.tensor([[(g if ip & 1 else -g), (g if ip & 2 else -g), (g if ip & 4 else -g)] for ip in range(8)],
                        dtype=torch.float64)


class _Ref:
    def __init__(self, p):
        self.dev = torch.device("cuda", DEVICE) if torch.cuda.is_available() else torch.device("cpu")
        as64 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=self.dev)  # noqa: E731
        self.n = p.n_dof
        self.conn = torch.as_tensor(p.conn, dtype=torch.long, device=self.dev)
        self.dofs = (3 * self.conn[:, :, None] + torch.arange(3, device=self.dev)).reshape(-1, 24)
        self.props = as64(p.props)
        X = as64(p.coords)[self.conn]  # [E, 8, 3]
        S, gp = _SIGN.to(self.dev), _gauss().to(self.dev)
        f = 1.0 + S[None] * gp[:, None, :]  # [ip, node, dir]
        dN = 0.125 * torch.stack([S[:, 0] * f[..., 1] * f[..., 2], S[:, 1] * f[..., 0] * f[..., 2],
                                  S[:, 2] * f[..., 0] * f[..., 1]], dim=-1)  # [ip, node, dir]
        J = torch.einsum("pad,eax->epdx", dN, X)
        self.w = torch.linalg.det(J)  # [E, 8]
        self.g = torch.einsum("epxd,pad->epax", torch.linalg.inv(J), dN)  # [E, ip, node, x]
        self.free = torch.ones(self.n, dtype=torch.float64, device=self.dev)
        self.free[torch.as_tensor(p.fixed, dtype=torch.long, device=self.dev)] = 0.0

    def lame(self, E=None, nu=None):
        E = self.props[:, 0] if E is None else E
        nu = self.props[:, 1] if nu is None else nu
        return E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))

    def b_matrix(self, lo, hi):
        """B of elements [lo, hi): [e, ip, 6, 24], engineering shear, xx yy zz xy yz zx."""
        g = self.g[lo:hi]
        B = torch.zeros(*g.shape[:2], 6, 8, 3, dtype=torch.float64, device=self.dev)
        for row, (i, j) in enumerate([(0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0)]):
            B[:, :, row, :, i] = g[..., j]
            if i != j:
                B[:, :, row, :, j] = g[..., i]
        return B.reshape(*g.shape[:2], 6, 24)

    def chunks(self, size=65536):
        E = self.conn.shape[0]
        return [(k, min(E, k + size)) for k in range(0, E, size)]

    def d_iso(self, lam, mu):
        D = torch.zeros(lam.shape[0], 6, 6, dtype=torch.float64, device=self.dev)
        D[:, :3, :3] = lam[:, None, None]
        for i in range(3):
            D[:, i, i] += 2 * mu
            D[:, 3 + i, 3 + i] = mu
        return D

    def element_matrices(self, D=None, E=None):
        """Ke [E, 24, 24] for the isotropic material or tangents D [E, 8, 6, 6]."""
        K = torch.empty(self.conn.shape[0], 24, 24, dtype=torch.float64, device=self.dev)
        lam, mu = self.lame(E)
        for lo, hi in self.chunks():
            B = self.b_matrix(lo, hi)
            Dc = self.d_iso(lam[lo:hi], mu[lo:hi])[:, None] if D is None else D[lo:hi]
            DB = (Dc @ B) * self.w[lo:hi, :, None, None]
            K[lo:hi] = B.reshape(hi - lo, 48, 24).transpose(1, 2) @ DB.reshape(hi - lo, 48, 24)
        return K

    def apply(self, K, x):
        """sum_e K_e x_e for x [n] or [n, k]."""
        y = torch.zeros_like(x)
        single = x.dim() == 1
        for lo, hi in self.chunks(1 << 19):
            d = self.dofs[lo:hi]
            xe = x[d]
            ye = (K[lo:hi] @ (xe[..., None] if single else xe))
            y.index_add_(0, d.reshape(-1), ye.reshape(-1) if single else ye.reshape(-1, x.shape[1]))
        return y

    def solve(self, K, b, fixed_values=None, rtol=1e-13, max_iter=20000):
        """K x = b on the free DOFs (x = 0 on the fixed ones) by Jacobi-CG; b [n] or [n, k]."""
        single = b.dim() == 1
        B = (b[:, None] if single else b) * self.free[:, None]
        diag = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        diag.index_add_(0, self.dofs.reshape(-1), torch.diagonal(K, dim1=1, dim2=2).reshape(-1))
        M = (self.free / diag)[:, None]
        x = torch.zeros_like(B)
        bn = torch.linalg.vector_norm(B, dim=0).clamp_min(1e-300)
        for _ in range(2):  # a second run from the true residual takes what rounding left
            r = B - self.apply(K, x) * self.free[:, None]
            p = torch.zeros_like(r)
            rz_old = torch.ones(B.shape[1], dtype=torch.float64, device=self.dev)
            for it in range(max_iter):
                z = M * r
                rz = (r * z).sum(0)
                p = z if it == 0 else z + (rz / rz_old.clamp_min(1e-300)) * p
                q = self.apply(K, p[:, 0] if single else p).reshape(p.shape) * self.free[:, None]
                a = rz / (p * q).sum(0).clamp_min(1e-300)
                x = x + a * p
                r = r - a * q
                rz_old = rz
                if it % 25 == 24 and bool((torch.linalg.vector_norm(r, dim=0) <= rtol * bn).all()):
                    break
        return x[:, 0] if single else x

    def strain(self, u):
        """Gauss-point strain [E, 8, 6]."""
        out = torch.empty(self.conn.shape[0], 8, 6, dtype=torch.float64, device=self.dev)
        for lo, hi in self.chunks():
            out[lo:hi] = torch.einsum("epsk,ek->eps", self.b_matrix(lo, hi), u[self.dofs[lo:hi]])
        return out

    def stress_iso(self, u):
        lam, mu = self.lame()
        return torch.einsum("est,ept->eps", self.d_iso(lam, mu), self.strain(u))

    def internal(self, sig):
        f = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        for lo, hi in self.chunks():
            fe = torch.einsum("epsk,eps,ep->ek", self.b_matrix(lo, hi), sig[lo:hi], self.w[lo:hi])
            f.index_add_(0, self.dofs[lo:hi].reshape(-1), fe.reshape(-1))
        return f

    def nodal(self, sig):
        """Gauss-point values extrapolated to the nodes, averaged over the elements at a node."""
        S, gp = _SIGN.to(self.dev), _gauss().to(self.dev)
        A = 0.125 * torch.prod(1.0 + S[None] * gp[:, None, :], dim=-1)  # [ip, node]
        v = torch.einsum("ap,eps->eas", torch.linalg.inv(A), sig)
        s = torch.zeros(self.n // 3, 6, dtype=torch.float64, device=self.dev)
        c = torch.zeros(self.n // 3, dtype=torch.float64, device=self.dev)
        s.index_add_(0, self.conn.reshape(-1), v.reshape(-1, 6))
        c.index_add_(0, self.conn.reshape(-1), torch.ones(v.shape[0] * 8, dtype=torch.float64, device=self.dev))
        return s / c[:, None]

    def j2(self, de, sig_n, ep_n):
        """Radial return, linear isotropic hardening: (stress, equivalent plastic strain, tangent)."""
        E, nu, sy, H = (self.props[:, k, None] for k in range(4))
        lam, G = self.lame()
        De = self.d_iso(lam, G)[:, None]
        st = sig_n + (De @ de[..., None])[..., 0]
        m = torch.tensor([1.0, 1, 1, 0, 0, 0], dtype=torch.float64, device=self.dev)
        p = st[..., :3].mean(-1)
        s = st - p[..., None] * m
        twice = 2.0 - m
        norm = torch.sqrt((twice * s * s).sum(-1))
        q = math.sqrt(1.5) * norm
        f = q - (sy + H * ep_n)
        G = G[:, None]
        plastic = f > 0
        dg = torch.where(plastic, f / (3 * G + H), torch.zeros_like(f))
        safe = torch.where(plastic, q, torch.ones_like(q))
        th1 = 1 - 3 * G * dg / safe
        sig = th1[..., None] * s + p[..., None] * m
        n = s / torch.where(plastic, norm, torch.ones_like(norm))[..., None]
        thb = 3 * G / (3 * G + H) - (1 - th1)
        Kb = E / (3 * (1 - 2 * nu))
        diag = torch.diag(1.0 / twice)  # 1 on the normal, 1/2 on the engineering-shear components
        Dp = (2 * G * th1)[..., None, None] * diag + (Kb - 2 * G * th1 / 3)[..., None, None] * torch.outer(m, m) \
            - (2 * G * thb)[..., None, None] * (n[..., :, None] * n[..., None, :])
        D = torch.where(plastic[..., None, None], Dp, De.expand(Dp.shape))
        return sig, ep_n + dg, D


def _von_mises(s):
    p = s[..., :3].mean(-1, keepdim=True)
    d = s[..., :3] - p
    j2 = 0.5 * (d * d).sum(-1) + (s[..., 3:] ** 2).sum(-1)
    return torch.sqrt(3.0 * j2)


def _face_load(p, faces, ref):
    """Per face of the regular x = max side: (t - q n) A / 4 on each of its four nodes."""
    elem, _, t, q = faces
    loc = np.array([1, 5, 6, 2])
    nodes = p.conn[elem][:, loc]
    X = p.coords[nodes]
    area = np.linalg.norm(np.cross(X[:, 1] - X[:, 0], X[:, 3] - X[:, 0]), axis=1)
    load = (t - q[:, None] * np.array([1.0, 0.0, 0.0])) * (area / 4.0)[:, None]
    f = np.zeros((p.n_nodes, 3))
    for a in range(4):
        np.add.at(f, nodes[:, a], load)
    return torch.as_tensor(f.ravel(), dtype=torch.float64, device=ref.dev)


def exact(case, seed):
    kind = case["kind"]
    p = _problem(case, seed)
    ref = _Ref(p)
    as64 = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=ref.dev)  # noqa: E731
    fixed = torch.as_tensor(p.fixed, dtype=torch.long, device=ref.dev)
    if kind in ("linear", "multigrid"):
        x = ref.solve(ref.element_matrices(), as64(p.f))
        return x.cpu().numpy() if case.get("buffers") == "host" else x
    if kind == "block":
        return ref.solve(ref.element_matrices(), as64(p.meta["F"].T)).T.contiguous()
    if kind == "design":
        r = _rng(seed, 7)
        rho = as64(p.meta["rho"])
        trial = as64(np.clip(p.meta["rho"] + 0.02 * r.standard_normal(p.n_elems), 0.3, 1.0))
        F = (as64(p.meta["F"]) * ref.free).T.contiguous()
        tip = 3 * int(p.meta["tip_node"]) + 2
        out = {}
        for key, d in (("", rho), ("trial_", trial)):
            E = E0 * d ** 3
            K = ref.element_matrices(E=E)
            U = ref.solve(K, F)
            out.update({key + "J1": (F * U).sum(), key + "J2": U[tip].sum(), key + "U": U.T.contiguous()})
            if key == "":
                dJ = F.clone()
                dJ[tip] += 1.0
                L = ref.solve(K, dJ)
                ue, le = U[ref.dofs], L[ref.dofs]
                g = -torch.einsum("eik,eik->e", le, K @ ue) / E
                out.update(g_rho=g * 3.0 * E0 * d ** 2, g_F=(U + L).T.contiguous())
        return out
    if kind == "newton":
        u = torch.zeros(p.n_dof, dtype=torch.float64, device=ref.dev)
        sig_n = torch.zeros(p.n_elems, 8, 6, dtype=torch.float64, device=ref.dev)
        ep_n = torch.zeros(p.n_elems, 8, dtype=torch.float64, device=ref.dev)
        u_n = u.clone()
        for step in (*_COMMITTED, _INCREMENT):
            target = as64(_target(p, step))
            for it in range(25):
                sig, ep, D = ref.j2(ref.strain(u - u_n), sig_n, ep_n)
                fint = ref.internal(sig)
                r = -fint * ref.free
                if it > 0 and float(torch.linalg.vector_norm(r)) <= 1e-11 * float(torch.linalg.vector_norm(fint)):
                    break
                K = ref.element_matrices(D=D)
                if it == 0:  # the prescribed values move first, with the tangent's response
                    du = torch.zeros_like(u)
                    du[fixed] = target - u[fixed]
                    r = r - ref.apply(K, du) * ref.free
                    u = u + du
                u = u + ref.solve(K, r, rtol=1e-11)
            u_n, sig_n, ep_n = u.clone(), sig, ep
        return u
    if kind == "assemble":
        x = as64(_direction(p, seed))
        K = ref.element_matrices()
        out = []
        for v in (x, x.float().double()):
            y = ref.apply(K, v * ref.free) * ref.free
            y[fixed] = v[fixed]
            out.append(y)
        return tuple(out)
    faces = _loaded_faces(p, case, seed)
    f = _face_load(p, faces, ref)
    if kind == "post":
        u = as64(_displacement(p, seed))
        sig = ref.stress_iso(u)
        fint = ref.internal(sig)
        r = (f - fint) * ref.free
        nodal = ref.nodal(sig)
        return {"f": f, "fint": fint, "r": r, "rnorm": torch.linalg.vector_norm(r),
                "fint_norm": torch.linalg.vector_norm(fint), "sigma": sig, "von_mises": _von_mises(sig),
                "nodal": nodal, "nodal_von_mises": _von_mises(nodal), "reactions": fint[fixed] - f[fixed]}
    u = ref.solve(ref.element_matrices(), f)
    sig = ref.stress_iso(u)
    fint = ref.internal(sig)
    host = lambda t: t.cpu().numpy()  # noqa: E731
    return {"u": host(u), "von_mises": host(_von_mises(sig)), "nodal": host(ref.nodal(sig)),
            "reactions": host(fint[fixed] - f[fixed])}
