"""The iteration kernels give the same bits every time, also around the points
where a run stops, replaces its residual and goes on: block 0 records a stop
while other blocks of the same kernel may still be starting."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,precision", [((96, 64, 64), "FP64"), ((128, 96, 96), "FP64"), ((96, 64, 64), "FP32_REFINE"),
                                             ((128, 96, 96), "FP32_REFINE")])
def test_solves_repeat_bit_for_bit(pkg, shape, precision):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=4)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64 | pkg.BUILD_FP32_ROUNDED | pkg.BUILD_SYMMETRIC)
    b = pkg.lifted_rhs(m, p.f)
    # a tolerance near the rounding of ||b - K x||: the recursive residual meets
    # it several times before the true one does
    a = pkg.SolverAlgo(tolerance=1e-10, precision_mode=getattr(pkg, "PRECISION_" + precision), max_iter=20000)
    first = None
    for _ in range(12):
        u, st = m.solve(b, a)
        now = (st.niter, st.n_refine, m.residual_history(), u)
        if first is None:
            first = now
            continue
        assert now[:2] == first[:2]
        assert np.array_equal(now[2], first[2]) and np.array_equal(now[3], first[3])
    m.close()


@pytest.mark.parametrize("shape,cycle", [((32, 16, 16), "FP64"), ((64, 32, 32), "FP32_REFINE"), ((128, 64, 64), "FP32_REFINE")])
def test_multigrid_solves_repeat_bit_for_bit(pkg, shape, cycle):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=5)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64 | pkg.BUILD_SYMMETRIC)
    m.mg_setup(*shape, precision=getattr(pkg, "PRECISION_" + cycle))
    b = pkg.lifted_rhs(m, p.f)
    a = pkg.SolverAlgo(tolerance=1e-10, precond_type=pkg.SOLV_PREC_MG, max_iter=500)
    first = None
    for _ in range(8):
        u, st = m.solve(b, a)
        now = (st.niter, m.residual_history(), u)
        if first is None:
            first = now
        assert now[0] == first[0] and np.array_equal(now[1], first[1]) and np.array_equal(now[2], first[2])
    m.close()
