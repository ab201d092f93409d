"""The one-kernel Jacobi-PCG of small FP64 systems against the chain of kernels
(the instrumented solve runs that chain on any size) and the oracle.

Sizes are node counts around the edges of its forms: a slice is 32 rows, up to
4 slices run in one CTA, up to 48 in a cluster of at most 16 CTAs.  The boxes
are compact: Jacobi-PCG does not solve long strips (condition number of order
length^4) to 1e-10 on either path.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# slices of 32 rows:      1        1 (full)   2          4 (full)   5          5
SHAPES = [(1, 1, 1), (7, 1, 1), (4, 2, 2), (7, 3, 3), (8, 3, 3), (9, 3, 3),
          # 16 (full)  17          48          48 (full)    49           51
          (7, 7, 7), (16, 3, 7), (8, 12, 12), (15, 11, 7), (7, 13, 13), (16, 11, 7)]


def _solve(pkg, m, b, **kw):
    return m.solve(b, pkg.SolverAlgo(tolerance=1e-10, **kw), raise_on_not_converged=False)


@pytest.mark.parametrize("shape", SHAPES)
def test_matches_the_kernel_chain(pkg, orc, shape):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=11)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64)
    b = pkg.lifted_rhs(m, p.f)
    u, st = _solve(pkg, m, b)
    h = m.residual_history()
    small = (p.n_nodes + 31) // 32 <= 48
    # one launch per run of the iterations, and a handful around it
    assert (m.last_timing()["kernel_launches"] < 3 * st.niter) == small or st.niter < 16
    m.set_instrument(True)
    v, sv = _solve(pkg, m, b)
    g = m.residual_history()
    m.set_instrument(False)
    assert st.converged and sv.converged and abs(st.niter - sv.niter) <= 2 + sv.niter // 100
    # both histories are those of the same recurrence: rounding grows along it
    k = min(10, h.size, g.size)
    ok = g[:k] > 1e-12 * g[0]
    np.testing.assert_allclose(h[:k][ok], g[:k][ok], rtol=1e-8)
    ref, _ = orc.Model(p).solve_linear(rtol=1e-13)
    assert np.linalg.norm(u - ref) <= 1e-9 * np.linalg.norm(ref)
    assert np.linalg.norm(v - ref) <= 1e-9 * np.linalg.norm(ref)
    m.close()


@pytest.mark.parametrize("shape", [(10, 2, 2), (15, 7, 7)])
def test_chunks_limits_and_starts(pkg, shape):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=12)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64)
    b = pkg.lifted_rhs(m, p.f)
    u, st = _solve(pkg, m, b)
    # the same run in launches of 7 iterations: the same numbers
    c, sc = _solve(pkg, m, b, check_every=7)
    assert sc.niter == st.niter and np.array_equal(c, u)
    # an iteration limit inside and at the end of a launch
    for limit in (5, 7, 14):
        _, sl = _solve(pkg, m, b, max_iter=limit, check_every=7)
        assert sl.niter == limit and not sl.converged and sl.status == pkg.STATUS_NOT_CONVERGED
    # from the solution, from a perturbed one, and without a preconditioner
    _, s0 = m.solve(b, pkg.SolverAlgo(tolerance=1e-9, use_x0=1), x=u.copy())
    assert s0.converged and s0.niter == 0
    w, s1 = m.solve(b, pkg.SolverAlgo(tolerance=1e-10, use_x0=1), x=u * (1 + 1e-3))
    n, s2 = m.solve(b, pkg.SolverAlgo(tolerance=1e-10, precond_type=0))
    for v, s in ((w, s1), (n, s2)):
        assert s.converged and np.linalg.norm(v - u) <= 1e-7 * np.linalg.norm(u)
    # zero load: no iteration
    z, s3 = m.solve(np.zeros_like(b), pkg.SolverAlgo(tolerance=1e-10))
    assert s3.converged and s3.niter == 0 and not z.any()
    m.close()
