"""Nodes that no element names: free ones stay where they are, fixed ones take their
prescribed value, and neither disturbs the rest of the solve, whatever the device
memory held before.  Their rows of the exported matrix are empty."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _with_extra(pkg, p, at, fixed):
    """p with a node inserted at each position of `at` (positions in the new numbering)."""
    n = p.n_nodes + len(at)
    old = np.setdiff1d(np.arange(n), at)
    coords = np.full((n, 3), 0.5)
    coords[old] = p.coords
    dof = (3 * old[:, None] + np.arange(3)).ravel()
    f = np.zeros(3 * n)
    f[dof] = p.f
    fx, val = dof[p.fixed], p.fixed_values
    if fixed:
        extra = (3 * np.asarray(at)[:, None] + np.arange(3)).ravel()
        fx, val = np.concatenate([fx, extra]), np.concatenate([val, 0.25 + 0.125 * np.arange(extra.size)])
        o = np.argsort(fx)
        fx, val = fx[o], val[o]
    return dataclasses.replace(p, coords=coords, conn=old[p.conn].astype(np.int32), fixed=fx.astype(np.int32),
                               fixed_values=val, f=f), dof


def _dirty_the_pool(pkg):
    """Freed device memory full of large numbers."""
    p = pkg.mesh.lognormal_cantilever(12, 6, 6, seed=1)
    p.props[:, 0] *= 1e300
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64 | pkg.BUILD_SYMMETRIC)
    m.close()


@pytest.mark.parametrize("shape", [(4, 2, 2), (9, 5, 4), (16, 11, 8)])
@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("at", [(0,), (31, 32), "last"])
def test_solves(pkg, shape, fixed, at):
    q = pkg.mesh.lognormal_cantilever(*shape, seed=8)
    at = (q.n_nodes,) if at == "last" else at
    p, dof = _with_extra(pkg, q, at, fixed)
    ref = pkg.FemModel.from_problem(q)
    ref.assemble(pkg.BUILD_FP64)
    want, _ = ref.solve(pkg.lifted_rhs(ref, q.f), pkg.SolverAlgo(tolerance=1e-12))
    ref.close()
    expect = np.zeros(p.n_dof)
    expect[dof] = want
    expect[p.fixed] = p.fixed_values
    for build, prec in ((pkg.BUILD_FP64, pkg.PRECISION_FP64),
                        (pkg.BUILD_FP64 | pkg.BUILD_SYMMETRIC, pkg.PRECISION_FP64),
                        (pkg.BUILD_FP64 | pkg.BUILD_FP32_ROUNDED | pkg.BUILD_SYMMETRIC, pkg.PRECISION_FP32_REFINE),
                        (pkg.BUILD_FP32, pkg.PRECISION_FP32_REFINE)):
        _dirty_the_pool(pkg)
        m = pkg.FemModel.from_problem(p)
        m.assemble(build)
        b = pkg.lifted_rhs(m, p.f, p.fixed_values)
        a = pkg.SolverAlgo(tolerance=1e-12, precision_mode=prec, max_iter=5000)
        u, st = m.solve(b, a)
        # two solutions with residuals of 1e-12 of the load: as close as the condition number (1e5) allows
        assert np.linalg.norm(u - expect) <= 1e-7 * np.linalg.norm(expect)
        extra = np.setdiff1d(np.arange(p.n_dof), dof)
        # a free one has a zero row and a zero load; the row of a fixed one is the
        # identity, and its residual part of the 1e-12 (twice: two evaluations of it)
        assert np.abs(u[extra] - expect[extra]).max() <= (2e-12 * np.linalg.norm(b) if fixed else 0.0)
        if prec == pkg.PRECISION_FP64:
            B = np.stack([b, 2 * b])
            X, _ = m.solve_block(B, pkg.SolverAlgo(tolerance=1e-12, max_iter=5000))
            assert np.linalg.norm(X - np.stack([expect, 2 * expect])) <= 1e-7 * np.linalg.norm(X)
            rp, c, v, _ = m.csr_export(index_base=0)
            assert (np.diff(rp)[extra] == 0).all() and np.isfinite(v).all()
        m.close()
