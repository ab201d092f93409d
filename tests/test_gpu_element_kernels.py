"""Assembly, internal forces, stresses and sensitivities at element and node
counts around the kernels' tile edges (32 rows per slice, 8 lanes per element,
4 elements per warp), on distorted, randomly numbered and high-valence meshes."""
import dataclasses

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _box(pkg, shape, seed, shuffle):
    """A distorted box with lognormal moduli, optionally numbered at random."""
    rng = np.random.default_rng(seed)
    p = pkg.mesh.lognormal_cantilever(*shape, seed=seed)
    h = p.coords.max(axis=0) / np.array(shape)
    p.coords += rng.uniform(-0.12, 0.12, p.coords.shape) * h
    if shuffle:
        new, elem = rng.permutation(p.n_nodes), rng.permutation(p.n_elems)
        coords = np.empty_like(p.coords)
        coords[new] = p.coords
        dof = (3 * new[:, None] + np.arange(3)).ravel()
        order = np.argsort(dof[p.fixed])
        f = np.empty_like(p.f)
        f[dof] = p.f
        p = dataclasses.replace(p, coords=coords, conn=np.ascontiguousarray(new[p.conn][elem].astype(np.int32)),
                                props=np.ascontiguousarray(p.props[elem]), fixed=dof[p.fixed][order].astype(np.int32),
                                fixed_values=p.fixed_values[order], f=f)
    return p


def _star(pkg, k):
    """k unit-size hexahedra that share one node and nothing else: its row has
    7 k + 1 blocks (they overlap in space, which the assembly does not notice)."""
    base, _ = pkg.mesh.box_mesh(1, 1, 1, 1.0, 1.0, 1.0)
    one = pkg.mesh.box_mesh(1, 1, 1, 1.0, 1.0, 1.0)[1][0]
    rng = np.random.default_rng(k)
    coords, conn = [np.zeros(3)], []
    for e in range(k):
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        q *= np.sign(np.linalg.det(q))  # a rotation
        x = (base + rng.uniform(-0.05, 0.05, base.shape)) @ q.T
        x -= x[0]
        ids = np.empty(8, np.int64)
        ids[0] = 0
        ids[1:] = len(coords) + np.arange(7)
        coords.extend(x[1:])
        conn.append(ids[one])
    coords, conn = np.array(coords), np.array(conn, np.int32)
    props = np.column_stack([rng.uniform(1e5, 3e5, k), np.full(k, 0.3)])
    n = 3 * coords.shape[0]
    fixed = np.array([0, 1, 2, 5, 40], np.int32)
    return pkg.mesh.Problem(f"star_{k}", (k, 1, 1), coords, conn, pkg.MAT_ELASTIC_ISO, props, fixed,
                            np.zeros(fixed.size), np.zeros(n))


MESHES = {
    "1": lambda pkg: _box(pkg, (1, 1, 1), 1, False),              # 8 nodes, 1 element
    "3": lambda pkg: _box(pkg, (3, 1, 1), 2, True),               # 16 nodes, 3 elements
    "7": lambda pkg: _box(pkg, (7, 1, 1), 3, False),              # 32 nodes
    "66 nodes": lambda pkg: _box(pkg, (10, 2, 1), 4, True),       # 20 elements
    "5x5x5": lambda pkg: _box(pkg, (5, 5, 5), 5, False),          # 216 nodes, 125 elements
    "9x7x6": lambda pkg: _box(pkg, (9, 7, 6), 6, True),           # 560 nodes, 378 elements
    "star 8": lambda pkg: _star(pkg, 8),                          # row of 57 blocks
    "star 13": lambda pkg: _star(pkg, 13),                        # 92, 99, 106 and 127 blocks: around the
    "star 14": lambda pkg: _star(pkg, 14),                        # longest row whose slice keeps its sums in
    "star 15": lambda pkg: _star(pkg, 15),                        # shared memory next to the coordinates
    "star 18": lambda pkg: _star(pkg, 18),
}


@pytest.mark.parametrize("mesh", MESHES)
def test_assembly(pkg, orc, mesh):
    p = MESHES[mesh](pkg)
    m = pkg.FemModel.from_problem(p)
    K = orc.Model(p).assemble()
    scale = np.abs(K.val).max()
    x = np.random.default_rng(0).standard_normal(p.n_dof)
    y = K.matvec(x)
    for build in (pkg.BUILD_FP64, pkg.BUILD_FP64 | pkg.BUILD_FP32,
                  pkg.BUILD_FP64 | pkg.BUILD_FP32_ROUNDED | pkg.BUILD_SYMMETRIC,
                  pkg.BUILD_FP64 | pkg.BUILD_SYMMETRIC):
        m.assemble(build)
        _, _, v, v32 = m.csr_export(values32=bool(build & (pkg.BUILD_FP32 | pkg.BUILD_FP32_ROUNDED)))
        # sums of up to 18 elements x 8 Gauss points of terms of the size of the
        # largest entry
        assert np.abs(v - K.val).max() <= 2e-13 * scale
        if build & pkg.BUILD_FP32_ROUNDED:
            assert np.array_equal(v32, v.astype(np.float32))
        elif build & pkg.BUILD_FP32:  # the same sums in 24 bits
            assert np.abs(v32 - K.val).max() <= 2e-5 * scale
        # the product of that storage: 81 to 381 terms a row
        assert np.abs(m.spmv(x) - y).max() <= 1e-12 * np.abs(y).max()
        if build & pkg.BUILD_FP32_ROUNDED:
            y32 = m.spmv(x.astype(np.float32), precision=pkg.PRECISION_FP32_REFINE)
            assert np.abs(y32 - y).max() <= 5e-5 * np.abs(y).max()
    m.close()


@pytest.mark.parametrize("mesh", MESHES)
def test_forces_and_sensitivities(pkg, orc, mesh):
    p = MESHES[mesh](pkg)
    m = pkg.FemModel.from_problem(p)
    rng = np.random.default_rng(1)
    u, lam = rng.standard_normal((2, p.n_dof)) * 1e-3
    o = orc.Model(p)
    f = m.internal_force(u)[0]
    ref = o.fint_elastic(u)
    assert np.abs(f - ref).max() <= 1e-12 * np.abs(ref).max()
    for U, L in ((u, lam), (np.stack([u, lam, u]), np.stack([lam, lam, u]))):
        g = m.adjoint_sensitivity(np.ascontiguousarray(U), np.ascontiguousarray(L))
        r = o.adjoint_dJdE(U.reshape(-1, p.n_dof), L.reshape(-1, p.n_dof))
        # one element's 24 x 24 form may cancel: relative to its largest terms
        assert np.abs(g - r).max() <= 1e-11 * np.abs(r).max()
    m.close()


@pytest.mark.parametrize("mesh", MESHES)
def test_uniform_strain(pkg, orc, mesh):
    """An affine displacement gives the same stress at every Gauss point and node."""
    p = MESHES[mesh](pkg)
    p.props[:] = p.props[0]
    m = pkg.FemModel.from_problem(p)
    G = np.random.default_rng(2).standard_normal((3, 3)) * 1e-3
    u = (p.coords @ G.T).ravel()
    e = np.array([G[0, 0], G[1, 1], G[2, 2], G[0, 1] + G[1, 0], G[1, 2] + G[2, 1], G[0, 2] + G[2, 0]])
    ref = orc.iso_D(*p.props[0]) @ e
    s, vm = m.stress(u)
    # gradients of distorted elements: condition of the Jacobian times rounding
    tol = 1e-11 * np.abs(ref).max()
    assert np.abs(s - _order(ref, s[0, 0])).max() <= tol
    ns, nvm = m.stress_nodal(u)
    assert np.abs(ns - _order(ref, s[0, 0])).max() <= tol
    d = ref[:3]
    v = np.sqrt(0.5 * ((d[0] - d[1])**2 + (d[1] - d[2])**2 + (d[2] - d[0])**2) + 3 * (ref[3:]**2).sum())
    assert np.abs(vm - v).max() <= tol and np.abs(nvm - v).max() <= tol
    m.close()


def _order(ref, got):
    """The shear components in the order that the library uses (xy, yz, xz or xy, xz, yz)."""
    alt = ref[[0, 1, 2, 3, 5, 4]]
    return ref if np.abs(got - ref).max() <= np.abs(got - alt).max() else alt


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 1), (6, 5, 3)])
@pytest.mark.parametrize("shuffle", [False, True])
def test_j2_tangent_is_the_derivative(pkg, shape, shuffle):
    """K v from the assembled J2 tangent against central differences of the
    internal force, far from the yield surface's kink."""
    q = _box(pkg, shape, 7, shuffle)
    sy, H = 250.0, 1000.0
    props = np.column_stack([np.full(q.n_elems, 200e3), np.full(q.n_elems, 0.3), np.full(q.n_elems, sy),
                             np.full(q.n_elems, H)])
    p = dataclasses.replace(q, mat_model_id=pkg.MAT_J2_ISO, props=props)
    m = pkg.FemModel.from_problem(p)
    rng = np.random.default_rng(3)
    # a strain of 1 % plus 10 % noise: every point at 5 to 10 times the yield strain
    G = np.diag([0.01, -0.004, -0.005])
    u = (p.coords @ G.T).ravel() + 1e-4 * rng.standard_normal(p.n_dof)
    v = rng.standard_normal(p.n_dof)
    v[p.fixed] = 0.0
    m.internal_force(u, update_state=True)
    for build in (pkg.BUILD_FP64, pkg.BUILD_FP64 | pkg.BUILD_SYMMETRIC):
        m.assemble(build)
        Kv = m.spmv(v)
        h = 1e-6
        d = (m.internal_force(u + h * v, update_state=False)[0] - m.internal_force(u - h * v, update_state=False)[0]) / (2 * h)
        free = np.ones(p.n_dof, bool)
        free[p.fixed] = False
        # h^2 of the third derivative (strain changes of 1e-4 of the strain), and
        # rounding 1e-16 / 1e-4
        assert np.abs(Kv - d)[free].max() <= 1e-5 * np.abs(d).max()
        m.internal_force(u, update_state=True)
    rp, col, val, _ = m.csr_export(index_base=0)
    K = sp.csr_matrix((val, col, rp), shape=(p.n_dof, p.n_dof))
    assert abs(K - K.T).max() <= 1e-12 * abs(K).max()
    m.close()
