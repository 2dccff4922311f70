"""Host calls in a process forked after its parent used the library's threads (smoothing, read-back)."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import ctypes as C, os, signal, sys, time
import numpy as np
import gubingluo_b200 as G

a = np.random.default_rng(0).random((200, 300)).astype(np.float32)
def smooth():
    b = a.copy()
    assert G.lib().rtm_velsmooth(b.ctypes.data_as(C.c_void_p), 200, 300, 3) == 0
    return b
if sys.argv[1] == "smoothing":
    want = smooth()
else:   # images of several copied chunks
    v = np.full((300, 600), 2000, np.float32)
    s = G.SurveyConfig(nx=600, nz=300, nt=20, dx=10.0, dz=10.0, dt=1e-3, npml=12, spx0=3000.0, spz0=20.0, mode=0)
    G.migrate(s, G.RunOptions(), [1], v, v)
    want = None
pid = os.fork()
if pid == 0:
    try:
        b = smooth()
        os._exit(0 if want is None or np.array_equal(b, want) else 3)
    finally:
        os._exit(4)
for _ in range(400):
    p, status = os.waitpid(pid, os.WNOHANG)
    if p:
        sys.exit(os.waitstatus_to_exitcode(status))
    time.sleep(0.05)
os.kill(pid, signal.SIGKILL)
os.waitpid(pid, 0)
sys.exit("the child hung")
"""


def _run(what):
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", SCRIPT, what], cwd=ROOT, capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr)


def test_smoothing_in_a_child_after_smoothing():
    _run("smoothing")


@pytest.mark.gpu
def test_smoothing_in_a_child_after_read_back():
    _run("read-back")
