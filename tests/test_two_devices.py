"""Contexts on two devices of one process, on a CUDA runtime without a GPU
(tests/host/fake_cudart.c, loaded before the library's): what is set up per device is
set up for each of them."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import ctypes
import numpy as np
from rheotool_gb300 import abi
from rheotool_gb300.case import SolverControl
from rheotool_gb300.mesh import channel_mesh
from rheotool_gb300.runtime import Context

fake = ctypes.CDLL(None)
mesh = channel_mesh(6, 9, 5)
N, F = mesh.nCells, mesh.nFaces
launches = []
for device in (0, 1):
    with Context(device) as ctx:
        ctx.upload_mesh(mesh)
        ctx.set_sweep(abi.SWEEP_SYSTOLIC)
        before = fake.fake_launches()
        # (a tolerance that nothing meets: one iteration, its sweeps launched)
        ctx.ldu_solve(np.ones(N), np.zeros(F), np.zeros(F), np.zeros((1, N)), np.zeros((1, N)),
                      SolverControl("PCG", "DIC", -1.0, 0.0, 0, 1))
        launches.append(fake.fake_launches() - before)
print(launches)
assert launches[0] == launches[1] > 0
"""


def test_sweeps_are_opted_in_on_each_device(tmp_path):
    cc = shutil.which("gcc") or shutil.which("cc")
    if cc is None:
        pytest.skip("no C compiler")
    from rheotool_gb300 import build
    build.build()
    fake = str(tmp_path / "libfakecudart.so")
    subprocess.check_call([cc, "-O1", "-fPIC", "-shared", "-o", fake, os.path.join(ROOT, "tests", "host", "fake_cudart.c")])
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env={**os.environ, "LD_PRELOAD": fake},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
