"""The V-cycle as an operator, over smoother degrees, precisions, box shapes,
level counts and coarsest solvers: symmetric, positive, and a solve with it
reaches the oracle's solution; refreshed hierarchies equal new ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

#        box           degree  coarse_max  levels
CASES = [((6, 4, 2), 1, 30, 0), ((10, 6, 6), 3, 0, 0), ((12, 8, 4), 2, 60, 0),
         ((20, 12, 12), 1, 0, 2), ((20, 12, 12), 3, 0, 2),  # coarsest 11 x 7 x 7 nodes: 1617 DOF, a Chebyshev solve
         ((24, 16, 16), 4, 200, 0), ((48, 32, 24), 2, 0, 0)]


def _model(pkg, shape, precision, degree, coarse_max, levels, symmetric):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=6)
    m = pkg.FemModel.from_problem(p)
    build = pkg.BUILD_FP64 | (pkg.BUILD_SYMMETRIC if symmetric else 0)
    m.assemble(build)
    m.mg_setup(*shape, degree=degree, coarse_max=coarse_max, max_levels=levels, precision=precision)
    return p, m, build


@pytest.mark.parametrize("shape,degree,coarse_max,levels", CASES)
@pytest.mark.parametrize("precision", ["FP64", "FP32_REFINE"])
@pytest.mark.parametrize("symmetric", [False, True])
def test_cycle(pkg, orc, shape, degree, coarse_max, levels, precision, symmetric):
    fp64 = precision == "FP64"
    p, m, build = _model(pkg, shape, getattr(pkg, "PRECISION_" + precision), degree, coarse_max, levels, symmetric)
    rng = np.random.default_rng(0)
    r1, r2 = rng.standard_normal((2, p.n_dof))
    r1[p.fixed] = r2[p.fixed] = 0.0
    z1, z2 = m.mg_apply(r1), m.mg_apply(r2)
    # M is symmetric up to the rounding of its precision, over some hundred
    # products in a row of levels and steps
    assert abs(z1 @ r2 - z2 @ r1) <= (1e-11 if fp64 else 2e-4) * np.linalg.norm(z1) * np.linalg.norm(r2)
    assert z1 @ r1 > 0 and z2 @ r2 > 0
    assert np.array_equal(m.mg_apply(r1), z1)
    a = pkg.SolverAlgo(tolerance=1e-10, precond_type=pkg.SOLV_PREC_MG, max_iter=500)
    b = pkg.lifted_rhs(m, p.f)
    u, st = m.solve(b, a)
    K = orc.Model(p).assemble()
    assert st.converged and np.linalg.norm(b - K.matvec(u)) <= 2e-10 * np.linalg.norm(b)
    # the values change: the hierarchy follows, and the kept graph with it
    p.props[:, 0] *= rng.uniform(0.5, 2.0, p.n_elems)
    m.set_material(p.mat_model_id, p.props)
    m.assemble(build)
    v, sv = m.solve(b, a)
    K = orc.Model(p).assemble()
    assert sv.converged and np.linalg.norm(b - K.matvec(v)) <= 2e-10 * np.linalg.norm(b)
    n = pkg.FemModel.from_problem(p)
    n.assemble(build)
    n.mg_setup(*shape, degree=degree, coarse_max=coarse_max, max_levels=levels,
               precision=getattr(pkg, "PRECISION_" + precision))
    w, sw = n.solve(b, a)
    assert sw.niter == sv.niter and np.array_equal(v, w)
    m.close()
    n.close()
