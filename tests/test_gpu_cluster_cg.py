"""The CG of a small grid in one cluster kernel equals the launched kernels bit for bit
(solution and iteration count): even and odd row lengths, more and fewer virtual blocks
than CTAs, both precisions, one to three sweeps a side, a solve stopped at its cap and a
start that is already converged.  GB2D_CLUSTER_CG=0, read once per process, selects the
launched kernels, hence the child processes."""
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
sys.path.insert(0, {root!r})
from tests.golden.cases import bubbles_case
gb = importlib.import_module("2d_engine_gb300")
out = {{}}
for ni, nj in ((64, 64), (33, 65), (97, 70), (128, 128), (130, 126), (24, 200)):
    ym = (nj - 1) / (ni - 1)
    case = bubbles_case(ni, nj, seed=ni + nj, x_max=1.0, y_max=ym)
    c = gb.Context(ni, nj, x_max=1.0, y_max=ym)
    for f, k in ((gb.FIELD_PHI, "phi"), (gb.FIELD_U, "u"), (gb.FIELD_V, "v")):
        c.set(f, case[k])
    rhs = c.poisson_assemble(0.5 / (ni - 1))[3]
    for prec in (gb.PRECISION_FP64, gb.PRECISION_MIXED):
        for nu, tol, cap in ((1, 1e-8, 2000), (2, 1e-9, 2000), (3, 1e-8, 2000), (2, 1e-12, 3)):
            x, st = c.poisson_solve(rhs, opts=gb.solve_opts(precision=prec, tolerance=tol, max_iterations=cap, mg_smooth=nu),
                                    allow_max_iters=True)
            key = f"{{ni}}x{{nj}}_{{prec}}_{{nu}}_{{cap}}"
            out[key] = x
            out[key + "_n"] = np.array([st.iterations, st.outer_iterations])
            x2, st2 = c.poisson_solve(rhs, x0=x, opts=gb.solve_opts(precision=prec, tolerance=1e-3, mg_smooth=nu))
            out[key + "_warm"] = np.append(x2.ravel(), st2.iterations)
    c.close()
np.savez({path!r}, **out)
"""


def run(path, launched):
    env = {k: v for k, v in os.environ.items() if k != "GB2D_CLUSTER_CG"}
    if launched:
        env["GB2D_CLUSTER_CG"] = "0"
    r = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, path=str(path))], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return np.load(path)


def test_cluster_cg_equals_launched_kernels(gb, tmp_path):
    a, b = run(tmp_path / "cluster.npz", False), run(tmp_path / "launched.npz", True)
    assert len(a.files) == 6 * 2 * 4 * 3
    for k in a.files:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
