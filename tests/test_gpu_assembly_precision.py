"""How far the displacements of the assembled FP64 stiffness are from those of the
exact one, on slender boxes, where a small error of one sign in every element (the
response of an element to a rigid translation) acts like an elastic foundation.

The reference is the stiffness in 80-bit arithmetic, solved to its precision.  The
tolerance: each row's response to a translation may be off by one unit in the last
place of its diagonal entry, of random sign; the error that this makes in the
displacements has a rounding's spread, computed here for each box, and four times
that is allowed.  Element errors that do not average out come to 5 to 60 times."""
import dataclasses

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sl

pytestmark = pytest.mark.gpu
L = np.longdouble


def _exact_elements(X, E, nu):
    X, E, nu = X.astype(L), E.astype(L), nu.astype(L)
    s = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], L)
    lam, mu = E * nu / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    K = np.zeros((len(E), 24, 24), L)
    for q in s / np.sqrt(L(3)):
        f = 1 + s * q
        d = np.stack([s[:, 0] * f[:, 1] * f[:, 2], s[:, 1] * f[:, 0] * f[:, 2], s[:, 2] * f[:, 0] * f[:, 1]], 1) / 8
        J = np.einsum("ai,eaj->eij", d, X)
        c = np.empty_like(J)
        for i in range(3):
            for j in range(3):
                a, b, k, m = (i + 1) % 3, (i + 2) % 3, (j + 1) % 3, (j + 2) % 3
                c[:, i, j] = J[:, a, k] * J[:, b, m] - J[:, a, m] * J[:, b, k]
        det = np.einsum("ej,ej->e", J[:, 0], c[:, 0])
        G = np.einsum("ai,eij->eaj", d, c) / det[:, None, None]
        t = np.einsum("eai,ebj->eaibj", G, G)
        dot = np.einsum("eai,ebi->eab", G, G)
        iso = np.swapaxes(t, 2, 4) + dot[:, :, None, :, None] * np.eye(3, dtype=L)[None, None, :, None, :]
        w = det[:, None, None, None, None]
        K += (w * (lam[:, None, None, None, None] * t + mu[:, None, None, None, None] * iso)).reshape(-1, 24, 24)
    return K


def _csr(p, Ke):
    n = p.n_dof
    dof = (3 * p.conn[:, :, None].astype(np.int64) + np.arange(3)).reshape(-1, 24)
    key = (np.repeat(dof, 24, 1) * n + np.tile(dof, (1, 24))).ravel()
    o = np.argsort(key, kind="stable")
    st = np.flatnonzero(np.r_[True, np.diff(key[o]) != 0])
    r, c, v = key[o][st] // n, key[o][st] % n, np.add.reduceat(Ke.ravel()[o], st)
    fixed = np.zeros(n, bool)
    fixed[p.fixed] = True
    m = fixed[r] | fixed[c]
    v = np.where(m & (r == c), L(1), np.where(m, L(0), v))
    return r, c, v


def _box(pkg, shape, uniform):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=4)
    if uniform:
        p.props[:, 0] = p.props[0, 0]
    return p


def _beside_a_star(pkg, p, k=13):
    """p and, apart from it, k fixed hexahedra around one node: a row of 92 blocks,
    with which the whole mesh is assembled by the kernel for long rows."""
    x0, e0 = pkg.mesh.box_mesh(1, 1, 1, 1.0, 1.0, 1.0)
    rng = np.random.default_rng(0)
    coords, conn = [np.zeros(3)], []
    for _ in range(k):
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        x = x0 @ (q * np.sign(np.linalg.det(q))).T
        ids = np.r_[0, len(coords) + np.arange(7)]
        coords.extend(x[1:] - x[0])
        conn.append(ids[e0[0]])
    n0 = p.n_nodes
    coords = np.array(coords) + 100.0
    return dataclasses.replace(
        p, coords=np.vstack([p.coords, coords]), conn=np.vstack([p.conn, n0 + np.array(conn)]).astype(np.int32),
        props=np.vstack([p.props, np.tile(p.props[:1], (k, 1))]),
        fixed=np.r_[p.fixed, 3 * n0 + np.arange(3 * len(coords))].astype(np.int32),
        fixed_values=np.r_[p.fixed_values, np.zeros(3 * len(coords))], f=np.r_[p.f, np.zeros(3 * len(coords))])


CASES = [(shape, uniform, form) for shape in [(40, 8, 8), (33, 5, 6)] for uniform in (False, True)
         for form in ("rows in registers", "long rows", "tangent")]


@pytest.mark.parametrize("shape,uniform,form", CASES)
def test_displacements(pkg, shape, uniform, form):
    p = _box(pkg, shape, uniform)
    if form == "long rows":
        p = _beside_a_star(pkg, p)
    E, nu, n = p.props[:, 0], p.props[:, 1], p.n_dof
    r, c, exact = _csr(p, _exact_elements(p.coords[p.conn], E, nu))
    rp = np.searchsorted(r, np.arange(n))
    lu = sl.splu(sp.csc_matrix((exact.astype(float), (r, c)), shape=(n, n)), permc_spec="MMD_AT_PLUS_A",
                 diag_pivot_thresh=0.0, options=dict(SymmetricMode=True))

    def solve(v):
        x = np.zeros(n, L)
        for _ in range(7):  # iterative refinement, residuals in 80 bits
            x = x + lu.solve((p.f.astype(L) - np.add.reduceat(v * x[c], rp)).astype(float))
        return x

    x = solve(exact)
    norm = float(np.sqrt((x * x).sum()))
    diag = exact[r == c].astype(float)
    diag[p.fixed] = 0.0
    rng = np.random.default_rng(0)
    spread = [np.linalg.norm(lu.solve(diag * x.astype(float) * rng.choice([-1.0, 1.0], n) * 2.0**-52)) for _ in range(8)]
    tol = 4 * np.sqrt(np.mean(np.square(spread)))

    if form == "tangent":  # at rest, where it is the elastic stiffness
        q = dataclasses.replace(p, mat_model_id=pkg.MAT_J2_ISO,
                                props=np.column_stack([E, nu, np.full(E.size, 1e3), np.full(E.size, 1e3)]))
    else:
        q = p
    m = pkg.FemModel.from_problem(q)
    if form == "tangent":
        m.internal_force(np.zeros(n), update_state=True)
    m.assemble(pkg.BUILD_FP64)
    _, col, val, _ = m.csr_export(index_base=0)
    m.close()
    assert np.array_equal(col, c)
    y = solve(val.astype(L))
    err = float(np.sqrt(((y - x) ** 2).sum()))
    assert err <= tol, (err / norm, tol / norm)
