"""The tiled mixed reinitialisation sweep evaluates the one-sided derivatives that a node's
update uses; it must equal the per-node kernel, which evaluates all four, bit for bit:
level sets with kinks, plateaus, exact zeros, noise and magnitudes outside FP32's range, on
grids at and beside the 32 x 8 tiles' edges.  The per-node kernel is chosen by an
environment variable that the library reads once, hence the child processes."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import importlib, sys
import numpy as np
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
from test_gpu_exact_sweeps import level_set
gb = importlib.import_module("2d_engine_gb300")
out = {{}}
for ni, nj in ((5, 9), (31, 8), (32, 16), (33, 17), (65, 41)):
    for kind in ("circles", "kink", "plateau", "noise", "large", "small"):
        for eps in (1e-6, 1e-20):
            phi, case = level_set(kind, ni, nj)
            c = gb.Context(ni, nj, weno_epsilon=eps, reinit_iterations=4, advection_precision=gb.PRECISION_MIXED)
            c.set(gb.FIELD_PHI, phi)
            c.reinitialization()
            out[f"{{ni}}x{{nj}}_{{kind}}_{{eps}}"] = c.get(gb.FIELD_PHI)
            c.close()
np.savez({path!r}, **out)
"""


def run(path, untiled):
    env = {k: v for k, v in os.environ.items() if k != "GB2D_REINIT_UNTILED"}
    if untiled:
        env["GB2D_REINIT_UNTILED"] = "1"
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, path=str(path))], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return np.load(path)


def test_selected_sides_equal_all_four(gb, tmp_path):
    a, b = run(tmp_path / "tiled.npz", False), run(tmp_path / "untiled.npz", True)
    assert len(a.files) == 60
    for k in a.files:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
