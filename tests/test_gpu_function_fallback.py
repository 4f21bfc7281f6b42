"""A stencil function whose staged grid cannot be described to TMA runs its
plain entry.  No grid that the library accepts is known to be one, so the test
links the compiled front end against an encoder that always fails."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from physis_gb300 import buildlib

pytestmark = pytest.mark.gpu

SHIM = r"""
#include "ps_internal.h"
namespace psg {
bool make_tmap_3d(CUtensorMap *, const GridView &, int, int) { return false; }
}
using namespace psg;
extern "C" __attribute__((visibility("default")))
int run(const char *source, const char *name, const float *host_in, float *host_out, int nx,
        int ny, int nz, int *staged) {
  JitKernel k;
  std::string err;
  if (!jit_compile(source, name, &k, &err)) return -1;
  *staged = (int)k.stages.size();
  const size_t pitch = ((size_t)nx * 4 + 127) / 128 * 128, rows = (size_t)ny * nz;
  GridView v[2] = {};
  int *dev_err = nullptr;
  if (cudaMalloc(&dev_err, 4) != cudaSuccess || cudaMemset(dev_err, 0, 4) != cudaSuccess) return -2;
  for (GridView &g : v) {
    void *p = nullptr;
    if (cudaMalloc(&p, pitch * rows) != cudaSuccess) return -2;
    if (cudaMemset(p, 0, pitch * rows) != cudaSuccess) return -2;
    g.ptr = p;
    g.pitch = pitch;
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.type = kFloat;
    g.esz = 4;
  }
  cudaMemcpy2D(v[0].ptr, pitch, host_in, nx * 4, nx * 4, rows, cudaMemcpyHostToDevice);
  const Box dom{{0, 0, 0}, {nx, ny, nz}};
  const cudaError_t e = jit_launch(k, dom, -1, v, nullptr, 148, dev_err, false, nullptr);
  if (e != cudaSuccess) return (int)e;
  if (cudaDeviceSynchronize() != cudaSuccess) return -3;
  cudaMemcpy2D(host_out, nx * 4, v[1].ptr, pitch, nx * 4, rows, cudaMemcpyDeviceToHost);
  jit_unload(&k);
  cudaFree(v[0].ptr);
  cudaFree(v[1].ptr);
  cudaFree(dev_err);
  return 0;
}
"""

SOURCE = """
void blur(const int x, const int y, const int z, PSGrid3DFloat g1, PSGrid3DFloat g2) {
  int nz = PSGridDim(g1, 2);
  float b = (z == 0) ? 0.0f : PSGridGet(g1, x, y, z - 1);
  float t = (z == nz - 1) ? 0.0f : PSGridGet(g1, x, y, z + 1);
  PSGridEmit(g2, PSGridGet(g1, x, y, z) + b + t);
}
"""


def test_plain_entry_without_a_tensor_map(tmp_path):
    buildlib.build()
    src, lib = tmp_path / "shim.cu", tmp_path / "libfallback.so"
    src.write_text(SHIM)
    subprocess.run([buildlib.nvcc(), "-shared"] + buildlib.common_flags()
                   + ["-o", str(lib), str(src), os.path.join(buildlib.BUILD, "jit.o"), "-ldl"],
                   check=True)
    L = ctypes.CDLL(str(lib))
    shape = (9, 21, 70)
    nz, ny, nx = shape
    a = np.random.default_rng(0).random(shape, dtype=np.float32)
    out, staged = np.zeros(shape, np.float32), ctypes.c_int(-1)
    f = lambda v: v.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    rc = L.run(SOURCE.encode(), b"blur", f(a), f(out), nx, ny, nz, ctypes.byref(staged))
    assert rc == 0 and staged.value == 1
    b, t = np.zeros_like(a), np.zeros_like(a)
    b[1:], t[:-1] = a[:-1], a[1:]
    assert np.array_equal(out, (a + b) + t)
