"""Every device-side CG loop ends by itself: its passes are capped whatever iteration limit
the caller gives (a kernel or graph launch cannot be left from the host).  Shown by reading
the two loops' limits: a run to the cap would take a GPU half a minute."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "2d_engine_gb300", "csrc")


def body(text, name):
    """The braces' content that follows the first definition of a kernel."""
    k = text.index("{", text.index(f"{name}(", text.index("__global__ void", text.index(name) - 400)))
    depth = 0
    for e in range(k, len(text)):
        depth += {"{": 1, "}": -1}.get(text[e], 0)
        if depth == 0:
            return text[k:e]


def test_device_loops_are_capped():
    text = open(os.path.join(CSRC, "gb2d_solver.cu")).read()
    cond = body(text, "k_loop_cond")
    assert re.search(r"n < pass_cap\(sc->max_it\)", cond)
    cluster = body(text, "k_cg_cluster")
    assert re.search(r"max_it = pass_cap\(g\.sc->max_it\)", cluster) and re.search(r"if \(it >= max_it\) break;", cluster)
    assert len(re.findall(r"->max_it", cond + cluster)) == 2  # no other use of the caller's limit


def test_cap_values(gb, tmp_path):
    import importlib
    b = importlib.import_module("2d_engine_gb300.build")
    src = tmp_path / "cap.cu"
    src.write_text('#include "gb2d_internal.cuh"\n#include <climits>\nusing gb2d::pass_cap;\n'
                   "static_assert(pass_cap(INT_MAX) == 1 << 20 && pass_cap((1 << 20) + 1) == 1 << 20 && pass_cap(1 << 20) == 1 << 20, \"\");\n"
                   "static_assert(pass_cap((1 << 20) - 1) == (1 << 20) - 1 && pass_cap(1) == 1 && pass_cap(0) == 0, \"\");\n")
    subprocess.run([b.nvcc(), "-std=c++17", *b.ARCH, "-I", os.path.join(ROOT, "include"), "-I", b.CSRC, "-c", str(src), "-o",
                    str(tmp_path / "cap.o")], check=True, timeout=200)
