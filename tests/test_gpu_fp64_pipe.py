"""The device forms of the FP64 products, quotients, roots and conversions on the
integer pipes (ttfld_fp64.cuh: carry chains, funnel shifts, the approximate
reciprocal instructions), on the operands of test_fp64_pipe.py, which tests the
host's forms: bit for bit the IEEE results."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_fp64_pipe import CSRC, boundary_quotients, operands, pairs, same

pytestmark = pytest.mark.gpu

SRC = r"""
#include "ttfld_fp64.cuh"
using namespace ttfld;
enum { MUL, DIV, ROOT, NARROW, WIDEN };
__global__ void run(int op, const void* a, const void* b, void* o, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double *x = (const double*)a, *y = (const double*)b;
    if (op == MUL) ((double*)o)[i] = mul_rn(x[i], y[i]);
    if (op == DIV) ((double*)o)[i] = div_rn(x[i], y[i]);
    if (op == ROOT) ((double*)o)[i] = sqrt_rn(x[i]);
    if (op == NARROW) ((float*)o)[i] = f32_rn(x[i]);
    if (op == WIDEN) ((double*)o)[i] = f64_of_f32(((const float*)a)[i]);
  }
}
// n elements of `in` bytes each in a and b (b may be null), of `out` bytes in o
extern "C" int device_op(int op, const void* a, const void* b, void* o, int n, int in, int out) {
  char *da = 0, *db = 0, *dz = 0;
  const size_t bytes = (size_t)n * in;
  int bad = cudaMalloc(&da, bytes) || cudaMalloc(&db, bytes) || cudaMalloc(&dz, (size_t)n * out);
  bad = bad || cudaMemcpy(da, a, bytes, cudaMemcpyHostToDevice);
  bad = bad || cudaMemcpy(db, b ? b : a, bytes, cudaMemcpyHostToDevice);
  if (!bad) run<<<304, 256>>>(op, da, db, dz, n);
  bad = bad || cudaDeviceSynchronize() || cudaMemcpy(o, dz, (size_t)n * out, cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(db);
  cudaFree(dz);
  return bad;
}
"""
MUL, DIV, ROOT, NARROW, WIDEN = range(5)


@pytest.fixture(scope="module")
def op(tmp_path_factory):
    from ttcode_gb300 import build
    d = tmp_path_factory.mktemp("fp64gpu")
    src, so = d / "t.cu", d / "t.so"
    src.write_text(SRC)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    f"-I{os.path.abspath(CSRC)}", str(src), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))

    def call(code, a, b=None, out=np.float64):
        a = np.ascontiguousarray(a)
        b = None if b is None else np.ascontiguousarray(b)
        o = np.empty(a.size, out)
        ptr = lambda v: None if v is None else v.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        assert lib.device_op(code, ptr(a), ptr(b), ptr(o), a.size, a.itemsize, o.itemsize) == 0
        return o
    return call


def test_products(op):
    a, b = pairs()
    with np.errstate(all="ignore"):
        same(op(MUL, a, b), a * b)


def test_quotients(op):
    with np.errstate(all="ignore"):
        for a, b in (pairs(), boundary_quotients()):
            same(op(DIV, a, b), a / b)


def test_roots(op):
    v, edge = operands()
    h = np.abs(v[60000:120000]).astype(np.float32).astype(np.float64)  # squares and their neighbours
    with np.errstate(all="ignore"):
        a = np.concatenate([np.abs(v), -np.abs(v[:10]), edge, h * h, np.nextafter(h * h, np.inf), np.nextafter(h * h, 0)])
        same(op(ROOT, a), np.sqrt(a))


def test_conversions(op):
    v, edge = operands()
    f = np.random.default_rng(3).integers(0, 1 << 32, 60000, dtype=np.uint64).astype(np.uint32).view(np.float32)
    with np.errstate(all="ignore"):
        ties = (f.astype(np.float64)[:20000] + np.nextafter(f, np.float32(0)).astype(np.float64)[:20000]) / 2
        a = np.concatenate([v, edge, f.astype(np.float64), ties])
        same(op(NARROW, a, out=np.float32), a.astype(np.float32))
        same(op(WIDEN, f), f.astype(np.float64))
