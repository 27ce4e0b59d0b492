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
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=40)
    assert r.returncode == 0, r.stderr
    return r.stdout.split()


def test_a_forked_child_has_its_own_memory():
    assert run(FORK) == ["parent", "True", "child", "0"]


CYCLES = """
import gc, sys, threading
sys.path.insert(0, "swalbe.jl_gb300")
from swalbe_gb300 import _results as R

R.release()
sys.setswitchinterval(1e-5)
gc.set_threshold(1)
sizes = [(2048, 2048 + i) for i in range(7)]  # up to seven unused mappings to look through


def work():
    for i in range(2000):
        cycle = [R.empty(sizes[i % 7])]
        cycle.append(cycle)  # dropped by the collector, wherever that runs
        a = R.empty(sizes[(i + 3) % 7])
        del cycle, a


ts = [threading.Thread(target=work) for _ in range(3)]
for t in ts:
    t.start()
for t in ts:
    t.join()
gc.set_threshold(700)
gc.collect()
R.release()
print("done", R._kept, len(R._free))
"""


def test_collector_inside_the_pool():
    """Arrays in reference cycles are given back by the garbage collector, also
    while this thread takes or gives back other memory."""
    assert run(CYCLES) == ["done", "0", "0"]


HELD = """
import os, signal, sys
sys.path.insert(0, "swalbe.jl_gb300")
from swalbe_gb300 import _results as R

R._lock.acquire()  # another thread is inside the pool when the process forks
pid = os.fork()
if pid == 0:
    signal.alarm(20)
    a = R.empty((2048, 2048))
    at = a.ctypes.data
    del a
    b = R.empty((2048, 2048))
    os._exit(0 if b.ctypes.data == at else 3)
print("child", os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]))
"""


def test_fork_while_another_thread_is_inside_the_pool():
    assert run(HELD) == ["child", "0"]
