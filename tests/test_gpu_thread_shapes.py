"""Threads that work on models of different row lengths at the same time: the
shared memory of a launch follows the model, and one model's launch must not
depend on what another thread has asked for in between."""
import dataclasses
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star(pkg, k):
    """k unit cubes around one node: its row has 1 + 7 k blocks."""
    x0, e0 = pkg.mesh.box_mesh(1, 1, 1, 1.0, 1.0, 1.0)
    rng = np.random.default_rng(0)
    coords, conn = [np.zeros(3)], []
    for _ in range(k):
        q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        x = x0 @ (q * np.sign(np.linalg.det(q))).T
        ids = np.r_[0, len(coords) + np.arange(7)]
        coords.extend(x[1:] - x[0])
        conn.append(ids[e0[0]])
    p = pkg.mesh.cantilever(1, 1, 1, 1.0, 1.0, 1.0, E=210e3)
    n = len(coords)
    return dataclasses.replace(p, coords=np.array(coords), conn=np.array(conn).astype(np.int32),
                               props=np.tile(p.props[:1], (k, 1)), fixed=np.arange(3, dtype=np.int32),
                               fixed_values=np.zeros(3), f=np.zeros(3 * n))


def _together(works, times):
    """Each work in its own thread, `times` times: its results, or the first exception of any."""
    got, bad = [[] for _ in works], []

    def loop(k):
        try:
            for _ in range(times):
                got[k].append(works[k]())
        except Exception as e:  # noqa: BLE001 (reported below)
            bad.append(e)

    ts = [threading.Thread(target=loop, args=(k,)) for k in range(len(works))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[0]
    return got


@pytest.mark.parametrize("form", ["elastic", "elastic fp32", "tangent"])
def test_assembly(pkg, form):
    models, works = [], []
    for p in (pkg.mesh.cantilever(1, 1, 1, 1.0, 1.0, 1.0, E=210e3), pkg.mesh.cantilever(4, 3, 3, 2.0, 1.0, 1.0, E=210e3),
              _star(pkg, 6), _star(pkg, 10), _star(pkg, 14)):
        if form == "tangent":
            p = dataclasses.replace(p, mat_model_id=pkg.MAT_J2_ISO, props=np.column_stack(
                [p.props[:, :2], np.full(p.n_elems, 1e3), np.full(p.n_elems, 1e3)]))
        m = pkg.FemModel.from_problem(p)
        if form == "tangent":
            m.internal_force(np.zeros(p.n_dof), update_state=True)
        models.append(m)
        build = pkg.BUILD_FP32 if form == "elastic fp32" else pkg.BUILD_FP64
        works.append(lambda m=m, build=build: m.assemble(build))
    _together(works, 300)
    for m in models:
        m.close()


def test_multigrid_set_up_and_block_solves(pkg):
    models, works = [], []
    for shape in ((4, 2, 2), (8, 4, 4), (8, 4, 12), (16, 8, 8)):
        p = pkg.mesh.lognormal_cantilever(*shape, seed=1)
        m = pkg.FemModel.from_problem(p)
        m.assemble(pkg.BUILD_FP64)
        models.append(m)
        B = np.outer(np.linspace(1.0, 2.0, 16), pkg.lifted_rhs(m, p.f))

        def work(m=m, B=B, shape=shape):
            m.mg_setup(*shape, coarse_max=30)
            X, _ = m.solve_block(B, pkg.SolverAlgo(tolerance=1e-8))
            return X

        works.append(work)
    alone = [w() for w in works]
    for ref, got in zip(alone, _together(works, 20)):
        for X in got:
            assert np.array_equal(X, ref)
    for m in models:
        m.close()
