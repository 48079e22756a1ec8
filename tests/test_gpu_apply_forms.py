"""The operator product's integer-pipe form has the plain form's bits: solutions, iteration
counts and a solve stopped after two iterations, on grids of 2^21 cells and more with even
and odd row lengths (two cells a thread and one).  GB2D_APPLY_INT=0, read once per process,
selects the plain form everywhere, hence the child processes."""
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
from test_gpu_cluster_tail import case_for, make
gb = importlib.import_module("2d_engine_gb300")
out = {{}}
for ni, nj in ((2048, 1024), (2049, 1025)):
    c = make(gb, case_for(ni, nj, 3), True)
    rhs = c.poisson_assemble(0.5 / (ni - 1))[3]
    for cap in (2, 2000):
        x, st = c.poisson_solve(rhs, opts=gb.solve_opts(precision=gb.PRECISION_MIXED, tolerance=1e-8, max_iterations=cap), allow_max_iters=True)
        out[f"{{ni}}_{{cap}}"] = x
        out[f"{{ni}}_{{cap}}_n"] = np.array([st.iterations, st.outer_iterations])
    c.close()
np.savez({path!r}, **out)
"""


def run(path, plain):
    env = {k: v for k, v in os.environ.items() if k != "GB2D_APPLY_INT"}
    if plain:
        env["GB2D_APPLY_INT"] = "0"
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, path=str(path))], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return np.load(path)


def test_integer_product_has_the_plain_products_bits(gb, tmp_path):
    a, b = run(tmp_path / "int.npz", False), run(tmp_path / "plain.npz", True)
    assert len(a.files) == 8 and a["2048_2_n"][0] == 2 and a["2048_2000_n"][0] > 5
    for k in a.files:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
