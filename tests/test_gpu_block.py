"""The multi-right-hand-side Jacobi-PCG: every number of threads per row, odd
meshes, right-hand sides that freeze early, and iteration limits inside and at
the end of a graph of iterations, against the oracle's matrix and the
single-right-hand-side solver."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _rhs(p, k, seed):
    rng = np.random.default_rng(seed)
    F = rng.standard_normal((k, p.n_dof))
    F[:, p.fixed] = 0.0
    return np.ascontiguousarray(F)


@pytest.mark.parametrize("shape", [(1, 1, 1), (7, 3, 1), (9, 5, 4)])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 7, 16, 17, 32])
def test_solutions(pkg, orc, shape, nrhs):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=8)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64)
    F = _rhs(p, nrhs, 1)
    if nrhs > 2:
        F[1] = 0.0  # solved before the first iteration
    X, st = m.solve_block(F, pkg.SolverAlgo(tolerance=1e-10))
    K = orc.Model(p).assemble()
    for k in range(nrhs):
        assert st[k].converged
        # the stop test's residual is 1e-10; the product's own rounding is far below
        assert np.linalg.norm(F[k] - K.matvec(X[k])) <= 2e-10 * np.linalg.norm(F[k])
    if nrhs > 2:
        assert st[1].niter == 0 and not X[1].any()
    m.close()


@pytest.mark.parametrize("nrhs", [1, 4, 16])
@pytest.mark.parametrize("limit", [1, 7, 32])
def test_iteration_limit(pkg, nrhs, limit):
    """x holds every counted iteration, wherever in a graph the run stops."""
    p = pkg.mesh.lognormal_cantilever(12, 7, 5, seed=9)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64)
    F = _rhs(p, nrhs, 2)

    def run(every):
        a = pkg.SolverAlgo(tolerance=1e-14, max_iter=limit, check_every=every)
        return m.solve_block(F, a, raise_on_not_converged=False)

    X, st = run(32)
    assert all(s.niter == limit and not s.converged for s in st)
    for every in (1, 5):
        Y, sy = run(every)
        assert np.array_equal(X, Y) and all(s.niter == limit for s in sy)
    # the same recurrence for one right-hand side alone: limit <= 32 steps of
    # rounding at 1e-16 each, amplified by the vectors' decay, stay below 1e-9
    u, _ = m.solve(F[0], pkg.SolverAlgo(tolerance=1e-14, max_iter=limit), raise_on_not_converged=False)
    assert np.linalg.norm(u - X[0]) <= 1e-9 * np.linalg.norm(u)
    m.close()


@pytest.mark.parametrize("shape,nrhs", [((48, 24, 24), 8), ((64, 40, 32), 32)])
def test_vectors_within_and_beyond_the_l2(pkg, shape, nrhs):
    """p, q and r of 18 and 204 MB: either side of the direction kernel's rule."""
    p = pkg.mesh.lognormal_cantilever(*shape, seed=8)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64)
    F = _rhs(p, nrhs, 3)
    X, st = m.solve_block(F, pkg.SolverAlgo(tolerance=1e-10))
    rp, col, val, _ = m.csr_export(index_base=0)
    K = sp.csr_matrix((val, col, rp), shape=(p.n_dof, p.n_dof))
    for k in range(nrhs):
        assert st[k].converged and np.linalg.norm(F[k] - K @ X[k]) <= 2e-10 * np.linalg.norm(F[k])
    m.close()
