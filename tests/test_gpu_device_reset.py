"""A process may end its CUDA context (cudaDeviceReset) and go on with new solvers: what
the library keeps for the process must not stand for what the context held."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes as C
import numpy as np
from shared_cfd_b200 import abi, cases, solver
from helpers import run_case

lib = solver.load_library()
runtime = C.CDLL("libcudart.so.12")  # the one the library has loaded
plate = cases.flat_plate(64, 40)
step = cases.reacting_step(scale=1.0 / 64.0, inner=3)
dual = cases.forward_step(0, n=8, scheme=abi.SCHEME_DUAL, viscous=1)
for case in (plate, step, dual):
    a = run_case(case, lib, 3)
    assert a["stats"].status == 0
    assert runtime.cudaDeviceReset() == 0
    b = run_case(case, lib, 3)
    assert b["stats"].status == 0
    assert np.array_equal(a["q"], b["q"])
print("same")
"""


@pytest.mark.parametrize("legacy", [False, True])
def test_solver_after_device_reset(gpu, legacy):
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests")]))
    env.pop("SCFD_SWEEP_LEGACY", None)
    if legacy:  # the generic residual and sweeps
        env["SCFD_SWEEP_LEGACY"] = "1"
    out = subprocess.run([sys.executable, "-c", PROGRAM], env=env, text=True, capture_output=True, timeout=300)
    assert out.returncode == 0 and out.stdout.endswith("same\n"), out.stdout + out.stderr
