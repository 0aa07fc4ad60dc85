"""The spectral kernels of a drop size in a process that has used no larger one: the first
2,048-node step asks k_setvelf for exactly 48 KiB of dynamic shared memory besides its static
variables, which needs the opt-in limit. A fresh process per size, since the limit stays set."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
from electricbubbles_gb300 import configs
from electricbubbles_gb300.api import Context
cfg = configs.single_drop(%d)
y = cfg.rku()
info = Context().rk2(cfg.nd, 1e-3, y, e0=0.5)
assert info["lap_ierr"] == 0 and info["stokes_ierr"] == 0
"""


@pytest.mark.parametrize("n", [1024, 2048, 4096])
def test_first_step_in_a_process(eblib, n):
    r = subprocess.run([sys.executable, "-c", CODE % n], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
