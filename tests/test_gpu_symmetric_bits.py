"""The assembled matrix is symmetric to the last bit in every precision, elastic and
J2, on regular, distorted, randomly numbered and high-valence meshes: the symmetric
storage, the full one and the exported CSR are the same matrix."""
import dataclasses

import numpy as np
import pytest
import scipy.sparse as sp

from test_gpu_element_kernels import MESHES, _box

pytestmark = pytest.mark.gpu

BOXES = {"16x7x5": ((16, 7, 5), False), "16x7x5 shuffled": ((16, 7, 5), True), "33x3x2": ((33, 3, 2), False)}


def _check(pkg, m, n):
    for build in (pkg.BUILD_FP64, pkg.BUILD_FP64 | pkg.BUILD_FP32,
                  pkg.BUILD_FP64 | pkg.BUILD_FP32_ROUNDED | pkg.BUILD_SYMMETRIC):
        m.assemble(build)
        w32 = bool(build & (pkg.BUILD_FP32 | pkg.BUILD_FP32_ROUNDED))
        rp, c, v, v32 = m.csr_export(index_base=0, values32=w32)
        for x in (v, v32) if w32 else (v,):
            K = sp.csr_matrix((x, c, rp), shape=(n, n))
            assert (K != K.T).nnz == 0
        if build & pkg.BUILD_SYMMETRIC:
            assert np.array_equal(v32, v.astype(np.float32))


@pytest.mark.parametrize("mesh", list(MESHES) + list(BOXES))
def test_elastic(pkg, mesh):
    p = MESHES[mesh](pkg) if mesh in MESHES else _box(pkg, BOXES[mesh][0], 9, BOXES[mesh][1])
    m = pkg.FemModel.from_problem(p)
    _check(pkg, m, p.n_dof)
    m.close()


@pytest.mark.parametrize("mesh", list(BOXES) + ["7", "66 nodes", "star 18"])
def test_j2_tangent(pkg, mesh):
    q = MESHES[mesh](pkg) if mesh in MESHES else _box(pkg, BOXES[mesh][0], 9, BOXES[mesh][1])
    props = np.column_stack([np.full(q.n_elems, 200e3), np.full(q.n_elems, 0.3), np.full(q.n_elems, 250.0),
                             np.full(q.n_elems, 1000.0)])
    p = dataclasses.replace(q, mat_model_id=pkg.MAT_J2_ISO, props=props)
    m = pkg.FemModel.from_problem(p)
    u = (p.coords @ np.diag([0.01, -0.004, -0.005])).ravel() + 1e-4 * np.random.default_rng(3).standard_normal(p.n_dof)
    m.internal_force(u, update_state=True)  # far past yield
    _check(pkg, m, p.n_dof)
    m.close()
