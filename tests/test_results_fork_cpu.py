"""Memory of large results across fork: a child's arrays and its parent's are
their own, whoever writes first and whoever takes memory again (no GPU)."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FORK = """
import os, sys
sys.path.insert(0, "swalbe.jl_gb300")
import numpy as np
from swalbe_gb300 import _results as R

held, dropped = R.empty((2048, 2048)), R.empty((2048, 2048))
held[...], dropped[...] = 1.0, 2.0
del dropped  # its memory is kept: both processes may take it
to_child, from_child = os.pipe(), os.pipe()
pid = os.fork()
if pid == 0:
    code = 1
    os.close(to_child[1])
    try:
        os.read(to_child[0], 1)  # the parent has written into its arrays
        ok = bool(np.all(held == 1.0))
        held[...] = 99.0
        taken = R.empty((2048, 2048))
        taken[...] = 5.0
        os.write(from_child[1], b"x")
        os.read(to_child[0], 1)
        ok = ok and bool(np.all(taken == 5.0)) and bool(np.all(held == 99.0))
        code = 0 if ok else 3
    finally:
        os._exit(code)
again = R.empty((2048, 2048))
again[...] = 6.0
del held
more = R.empty((2048, 2048))
more[...] = 7.0
os.write(to_child[1], b"x")
os.read(from_child[0], 1)
parent_ok = bool(np.all(again == 6.0)) and bool(np.all(more == 7.0))
os.write(to_child[1], b"x")
status = os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1])
print("parent", parent_ok, "child", status)
"""


def run(script):
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    return r.stdout.split()


def test_a_forked_child_has_its_own_memory():
    assert run(FORK) == ["parent", "True", "child", "0"]
