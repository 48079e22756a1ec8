"""The buffers that a context makes on first use (the adjoints', the general jump-Poisson
solve's) stand all or not at all.  The library's own object files are linked with a fake
allocator that fails at a chosen call: the failing call reports an error, leaves no pointer
and no memory behind, and the next call tries again instead of reporting success."""
import glob
import os
import subprocess

from conftest import ROOT

HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

#include "gb2d_internal.cuh"

static int g_calls, g_fail_at;
static std::map<void*, int> g_live;
static cudaError_t step() { return ++g_calls == g_fail_at ? cudaErrorMemoryAllocation : cudaSuccess; }
extern "C" {
cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
  cudaError_t e = step();
  if (e == cudaSuccess) g_live[*p = malloc(n)] = 1;
  return e;
}
cudaError_t __wrap_cudaMemset(void* p, int, size_t) { return g_live.count(p) ? step() : cudaErrorInvalidValue; }
cudaError_t __wrap_cudaStreamSynchronize(cudaStream_t) { return step(); }
cudaError_t __wrap_cudaFree(void* p) {
  if (!g_live.erase(p)) return cudaErrorInvalidValue;
  free(p);
  return cudaSuccess;
}
}

static int check(int (*make)(gb2d_ctx*), int buffers) {
  gb2d_ctx* clean = new gb2d_ctx();
  clean->grid.ni = 8;
  clean->grid.nj = 6;
  g_calls = g_fail_at = 0;
  gb2d_ctx* c = new gb2d_ctx(*clean);
  if (make(c) != GB2D_OK || (int)g_live.size() != buffers) return 1;
  const int steps = g_calls;
  g_live.clear();
  for (int k = 1; k <= steps; ++k) {
    memcpy((void*)c, (void*)clean, sizeof *c);
    g_calls = 0;
    g_fail_at = k;
    if (make(c) == GB2D_OK || !g_live.empty() || c->err[0] == 0) return printf("step %d of %d: %zu buffers left\n", k, steps, g_live.size()), 2;
    memset(c->err, 0, sizeof c->err);
    if (memcmp((void*)c, (void*)clean, sizeof *c)) return printf("step %d of %d: a pointer is left\n", k, steps), 3;
    g_calls = 0;
    if (make(c) == GB2D_OK) return printf("step %d of %d: the second call fails too, and must say so\n", k, steps), 4;
    g_calls = g_fail_at = 0;
    if (make(c) != GB2D_OK || (int)g_live.size() != buffers || g_calls != steps) return printf("step %d of %d: no recovery\n", k, steps), 5;
    g_live.clear();
  }
  return 0;
}

int main() {
  const int a = check(gb2d::adjoint_buffers, 10), b = check(gb2d::jump_buffers, 8);
  printf("adjoint %d jump %d\n", a, b);
  return a || b;
}
"""


def test_first_use_buffers_stand_all_or_not_at_all(gb, tmp_path):
    import importlib
    b = importlib.import_module("2d_engine_gb300.build")
    src, exe = tmp_path / "harness.cu", tmp_path / "harness"
    src.write_text(HARNESS)
    wrap = [f"-Xlinker=--wrap={f}" for f in ("cudaMalloc", "cudaMemset", "cudaStreamSynchronize", "cudaFree")]
    objs = sorted(glob.glob(os.path.join(b.OUT, "gb2d_*.o")))
    assert objs
    subprocess.run([b.nvcc(), "-std=c++17", *b.ARCH, "-I", os.path.join(ROOT, "include"), "-I", b.CSRC, *wrap, str(src), *objs, "-o", str(exe)],
                   check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
