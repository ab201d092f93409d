"""Newton increments on either side of the rule that gives the FP64 tangent the
symmetric storage: the equilibrium that the increment reports holds for the
matrix-free internal force, and the products afterwards are those of the
exported matrix."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,precond", [((48, 24, 24), "jacobi"), ((56, 28, 28), "jacobi"), ((57, 27, 29), "jacobi"),
                                           ((56, 28, 28), "mg"), ((88, 48, 48), "mg")])
def test_increment(pkg, shape, precond):
    p = pkg.mesh.j2_bar(*shape)
    m = pkg.FemModel.from_problem(p)
    kw = {}
    if precond == "mg":
        m.internal_force(np.zeros(p.n_dof))
        m.assemble(pkg.BUILD_FP64)
        m.mg_setup(*shape, precision=pkg.PRECISION_FP32_REFINE)
        kw["precond_type"] = pkg.SOLV_PREC_MG
    free = np.ones(p.n_dof, bool)
    free[p.fixed] = False
    for step in (1, 9):  # elastic, then plastic
        r = m.nr_increment(pkg.mesh.j2_bar_target(p, step), tolerance_force=1e-9,
                           lin=pkg.SolverAlgo(tolerance=1e-10, max_iter=20000, **kw))
        assert r.converged
        u = m.displacement()
        f = m.internal_force(u, update_state=False)[0]
        # tolerance_force times ||F_int||; the same sums in the same kernels
        assert np.linalg.norm(f[free]) <= 1.01e-9 * np.linalg.norm(f)
        m.commit()
    rp, col, val, _ = m.csr_export(index_base=0)
    K = sp.csr_matrix((val, col, rp), shape=(p.n_dof, p.n_dof))
    x = np.random.default_rng(3).standard_normal(p.n_dof)
    y = m.spmv(x)
    # K_ji for K_ij (each the sum of up to 8 elements x 8 Gauss points, up to 64
    # units of 1.1e-16 of its terms, which may cancel), then 81 products
    assert np.all(np.abs(y - K @ x) <= 1e-13 * (abs(K) @ np.abs(x)) + 1e-300)
    m.close()
