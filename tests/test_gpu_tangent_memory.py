"""The storage of the tangent in a Newton increment does not depend on how much
device memory is free at the moment: the same bits with plenty and with little,
and where the symmetric storage does not fit the increment runs on the full one.
Each case in a process of its own."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import sys
sys.path.insert(0, %r)
import numpy as np, torch
import __graft_entry__
pkg = __graft_entry__.load_package()

def increment(shape, leave_mib):
    # one increment past first yield; leave_mib: device memory that the caller leaves to it
    p = pkg.mesh.j2_bar(*shape)
    m = pkg.FemModel.from_problem(p)
    m.internal_force(np.zeros(p.n_dof), update_state=True)
    m.assemble(pkg.BUILD_FP64)
    torch.cuda.synchronize()
    hold = None
    if leave_mib:
        torch.zeros(1, device="cuda")
        free, _ = torch.cuda.mem_get_info()
        hold = torch.empty(free - (leave_mib << 20), dtype=torch.uint8, device="cuda")
    for step in (1, 9):
        r = m.nr_increment(pkg.mesh.j2_bar_target(p, step), tolerance_force=1e-9,
                           lin=pkg.SolverAlgo(tolerance=1e-10, max_iter=20000))
        assert r.converged
        m.commit()
    u = m.displacement()
    m.close()
    del hold
    torch.cuda.empty_cache()
    return u
""" % ROOT


def _run(body):
    r = subprocess.run([sys.executable, "-c", HEAD + textwrap.dedent(body)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]


def test_same_bits_with_little_memory_free():
    # full values of 93 MB, symmetric storage of some 80 MB: room for it in 330 MiB, not for four times the full values
    _run("""
    assert np.array_equal(increment((56, 28, 28), 0), increment((56, 28, 28), 330))
    """)


def test_goes_on_without_the_storage():
    # full values of 456 MB; the symmetric storage (some 380 MB) does not fit, the vectors (6 MB each) do
    _run("""
    u, v = increment((96, 48, 48), 0), increment((96, 48, 48), 150)
    # two runs to 1e-9 of the internal force
    assert np.linalg.norm(u - v) <= 1e-6 * np.linalg.norm(u)
    """)
