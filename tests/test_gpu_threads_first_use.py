"""Handles made by several threads at once in a process that has run no kernel
yet: each kernel's shared-memory limit is raised by the first caller that needs
it, and no other caller may launch the kernel before that is done (its launch
would be refused)."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import threading
import numpy as np
import mat3d_b200 as m3d
mode = %r
n = 8
gate = threading.Barrier(n)
out, err = [None] * n, []
phase2 = (np.arange(1024 * 16) %% 3 != 0).astype(np.int32)
phase3 = (np.arange(8 * 8 * 128) %% 3 != 0).astype(np.int32)
def work(i):
    try:
        gate.wait()
        if mode == "plane":
            s = m3d.Solver2D(1024, 16)
            s.material((3e9, 0.35, 70e9, 0.2), phase2)
            s.set_load([0.005, 0.0, 0.0])
            s.run(2)
            out[i] = s.fields()[0].copy()
        else:
            s = m3d.Solver(m3d.KIND_THERMAL, 8, 8, 128, precision="fp64")
            s.set_material_thermal(1.0, 5.0, phase3)
            s.set_load(np.array([0.1, 0.2, 1.0]))
            s.run(1e-8)
            out[i] = s.field().copy()
        s.close()
    except Exception as e:
        err.append(repr(e))
threads = [threading.Thread(target=work, args=(i,)) for i in range(n)]
[t.start() for t in threads]
[t.join() for t in threads]
assert not err, err
assert all(np.array_equal(o, out[0]) for o in out)
print("same")
"""


@pytest.mark.parametrize("mode", ["plane", "solver"])
def test_first_use_by_threads(mode):
    r = subprocess.run([sys.executable, "-c", SCRIPT % mode], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr
