"""Models opened, solved and closed by several threads at once share one memory
pool per device: each gets the numbers it gets alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [2, 5])
def test_threads(pkg, threads):
    shapes = [(10, 2, 2), (24, 12, 12), (7, 5, 3), (32, 16, 16), (16, 16, 16)][:threads]

    def run(shape):
        p = pkg.mesh.lognormal_cantilever(*shape, seed=3)
        m = pkg.FemModel.from_problem(p)
        m.assemble(pkg.BUILD_FP64 | pkg.BUILD_SYMMETRIC)
        u, st = m.solve(pkg.lifted_rhs(m, p.f), pkg.SolverAlgo(tolerance=1e-9))
        s, vm = m.stress(u)
        m.close()
        return st.niter, u, s, vm

    alone = [run(s) for s in shapes]
    got = [[] for _ in shapes]

    def work(k):
        for _ in range(4):
            got[k].append(run(shapes[k]))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(len(shapes))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k, ref in enumerate(alone):
        assert len(got[k]) == 4
        for r in got[k]:
            assert r[0] == ref[0] and all(np.array_equal(a, b) for a, b in zip(r[1:], ref[1:]))
