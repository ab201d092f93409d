"""The oracle's solves give the same bits on any number of threads and every time."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

BODY = """
import sys, hashlib
sys.path.insert(0, %r)
import __graft_entry__
pkg = __graft_entry__.load_package()
from oracle import oracle as O
p = pkg.mesh.lognormal_cantilever(24, 12, 12, seed=1)
for _ in range(2):
    u, _ = O.Model(p).solve_linear(rtol=1e-12)
    print(hashlib.sha256(u.tobytes()).hexdigest())
""" % ROOT


def test_solves_repeat_bit_for_bit():
    got = set()
    for threads in (1, 3, 8):
        r = subprocess.run([sys.executable, "-c", BODY], capture_output=True, text=True, timeout=300,
                           env=dict(os.environ, OMP_NUM_THREADS=str(threads), OMP_DYNAMIC="false"))
        assert r.returncode == 0, r.stderr[-2000:]
        got |= set(r.stdout.split())
    assert len(got) == 1
