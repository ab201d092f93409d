"""The matrix-free operators on meshes around and beyond the elements that their
scratch array holds (2^18), and the device memory they take."""
import dataclasses
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHAPES = [(64, 64, 64), (65, 64, 64), (132, 64, 64)]  # 2^18 elements, one plane more, three passes


def _problem(pkg, shape, shuffle):
    p = pkg.mesh.lognormal_cantilever(*shape, seed=2)
    if not shuffle:
        return p
    rng = np.random.default_rng(0)
    new, elem = rng.permutation(p.n_nodes), rng.permutation(p.n_elems)
    coords = np.empty_like(p.coords)
    coords[new] = p.coords
    dof = (3 * new[:, None] + np.arange(3)).ravel()
    f = np.empty_like(p.f)
    f[dof] = p.f
    return dataclasses.replace(p, coords=coords, conn=np.ascontiguousarray(new[p.conn][elem].astype(np.int32)),
                               props=np.ascontiguousarray(p.props[elem]), fixed=np.sort(dof[p.fixed]).astype(np.int32), f=f)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("shuffle", [False, True])
def test_forces(pkg, orc, shape, shuffle):
    p = _problem(pkg, shape, shuffle)
    u = np.random.default_rng(1).standard_normal(p.n_dof) * 1e-6
    ref = orc.Model(p).fint_elastic(u)
    m = pkg.FemModel.from_problem(p)
    f = m.internal_force(u)[0]
    # sums of 8 elements x 8 Gauss points
    assert np.abs(f - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.array_equal(f, m.internal_force(u)[0])
    m.close()
    # the J2 material below yield: the same forces
    q = dataclasses.replace(p, mat_model_id=pkg.MAT_J2_ISO, props=np.column_stack([p.props[:, :2], np.full(p.n_elems, 1e9),
                                                                                   np.full(p.n_elems, 1e3)]))
    m = pkg.FemModel.from_problem(q)
    g = m.internal_force(u)[0]
    assert np.abs(g - ref).max() <= 1e-12 * np.abs(ref).max()
    m.close()


@pytest.mark.parametrize("shape", SHAPES[1:])
def test_refined_residual(pkg, shape):
    """The refined solve takes its residual from the eliminated operator; the assembled matrix confirms it."""
    p = _problem(pkg, shape, False)
    p.fixed_values = np.linspace(0.0, 1e-6, p.fixed.size)
    m = pkg.FemModel.from_problem(p)
    m.assemble(pkg.BUILD_FP64 | pkg.BUILD_FP32_ROUNDED)
    b = pkg.lifted_rhs(m, p.f, p.fixed_values)
    u, st = m.solve(b, pkg.SolverAlgo(tolerance=1e-8, precision_mode=pkg.PRECISION_FP32_REFINE, max_iter=20000))
    r = b - m.spmv(u)
    # 1e-8 of the load, and the rounding of K u in either evaluation
    assert np.linalg.norm(r) <= 1.1e-8 * np.linalg.norm(b)
    assert np.abs(u[p.fixed] - p.fixed_values).max() <= 1.1e-8 * np.linalg.norm(b)
    m.close()


def test_scratch_does_not_grow_with_the_mesh():
    """5.7M elements: 192 bytes for each would be 1.1 GB, more than the pool keeps."""
    body = """
import sys
sys.path.insert(0, %r)
import torch
import __graft_entry__
pkg = __graft_entry__.load_package()
p = pkg.mesh.cantilever(224, 160, 160, 2.0, 1.0, 1.0, E=210e3)
m = pkg.FemModel.from_problem(p)
u = torch.rand(p.n_dof, dtype=torch.float64, device="cuda")
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
m.internal_force(u)
torch.cuda.synchronize()
took = (free - torch.cuda.mem_get_info()[0]) / 2**20
# the scratch (50 MB) and vectors of 140 MB: the caller's force and residual, the context's own
# (two or three); with 192 bytes per element it would come to 1.6 GB
assert took <= 900, took
m.close()
""" % ROOT
    r = subprocess.run([sys.executable, "-c", body], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
