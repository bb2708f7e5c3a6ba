"""The FP64 products, quotients, roots and conversions that the kernels form on
the integer pipes (ttfld_fp64.cuh), and the kernels' index division, compiled
for the host and compared with the machine's own arithmetic bit for bit: at
the ends of the exponent range, on zeros, infinities and NaN, on mantissas of
all ones, on quotients next to a rounding boundary, and on random operands.
The first FP32 guesses of the quotient and the root are also given the error
of the device's approximate instructions (3 ulp)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "ttcode_gb300", "csrc")

SRC = r"""
#include "ttfld_fp64.cuh"
using namespace ttfld;
extern "C" {
void t_mul(const double* a, const double* b, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = mul_rn(a[i], b[i]); }
void t_div(const double* a, const double* b, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = div_rn(a[i], b[i]); }
void t_root(const double* a, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = sqrt_rn(a[i]); }
void t_narrow(const double* a, float* o, long n) { for (long i = 0; i < n; ++i) o[i] = f32_rn(a[i]); }
void t_widen(const float* a, double* o, long n) { for (long i = 0; i < n; ++i) o[i] = f64_of_f32(a[i]); }
long t_index(int d, const unsigned* t, long n) {
  const FastDiv f = fast_div(d);
  long bad = 0;
  for (long i = 0; i < n; ++i) { unsigned r, q = div_rem(f, t[i], r); bad += q != t[i] / (unsigned)d || r != t[i] % (unsigned)d; }
  return bad;
}
}
"""


@pytest.fixture(scope="module", params=["0.0f", "3.6e-7f", "-3.6e-7f"])
def lib(request, tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64")
    src, so = d / "t.cpp", d / "t.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}",
                    f"-DTT_GUESS_ERROR(v)=((v)*(1.0f+{request.param}))", str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def call(fn, *arrays, out=np.float64):
    o = np.empty(arrays[0].size, out)
    fn(*[a.ctypes.data_as(ctypes.c_void_p) for a in arrays], o.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(o.size))
    return o


def same(got, want):
    w = np.uint64 if got.dtype == np.float64 else np.uint32
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(w), want[~nan].view(w))


def operands(n=60000):
    rng = np.random.default_rng(0)
    bits = rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2) + rng.integers(0, 2, n, dtype=np.uint64)
    mid = (bits & np.uint64(0x800FFFFFFFFFFFFF)) | (rng.integers(990, 1060, n, dtype=np.uint64) << np.uint64(52))
    ones = mid | np.uint64(0xFFFFFFFFFFFF0)
    few = mid & ~np.uint64(0xFFFFFFFFF0000)
    edge = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072014e-308, 2.225073858507201e-308,
                     1.7976931348623157e308, 1.0, -1.0, 2.0, 0.5, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1e-300, 1e300])
    return np.concatenate([a.view(np.float64) for a in (bits, mid, ones, few)]), edge


def pairs():
    v, edge = operands()
    rng = np.random.default_rng(1)
    w = rng.permutation(v)
    e1, e2 = (m.ravel() for m in np.meshgrid(edge, edge))
    mixed = rng.choice(edge, 4000)
    return (np.concatenate([v, e1, mixed, v[:4000]]), np.concatenate([w, e2, v[:4000], mixed]))


def boundary_quotients():
    """a, b with a/b within a few 2^-107 of half way between two doubles."""
    rng = np.random.default_rng(2)
    a, b = [], []
    for _ in range(3000):
        B = int(rng.integers(1 << 52, 1 << 53)) | 1
        for s in (53, 54):
            inv = pow(pow(2, s, B), -1, B)
            for t in (1, 2, -1, -2):
                A = inv * t % B + (B if s == 53 else 0)
                if 0 < A < 1 << 53:
                    a.append(float(A))
                    b.append(float(B))
    return np.array(a), np.array(b)


def test_products(lib):
    a, b = pairs()
    with np.errstate(all="ignore"):
        same(call(lib.t_mul, a, b), a * b)


def test_quotients(lib):
    with np.errstate(all="ignore"):
        for a, b in (pairs(), boundary_quotients()):
            same(call(lib.t_div, a, b), a / b)


def test_roots(lib):
    v, edge = operands()
    h = np.abs(v[60000:120000]).astype(np.float32).astype(np.float64)  # squares and their neighbours
    a = np.concatenate([np.abs(v), -np.abs(v[:10]), edge, h * h, np.nextafter(h * h, np.inf), np.nextafter(h * h, 0)])
    with np.errstate(all="ignore"):
        same(call(lib.t_root, a), np.sqrt(a))


def test_conversions(lib):
    v, edge = operands()
    f = np.random.default_rng(3).integers(0, 1 << 32, 60000, dtype=np.uint64).astype(np.uint32).view(np.float32)
    with np.errstate(all="ignore"):
        ties = (f.astype(np.float64)[:20000] + np.nextafter(f, np.float32(0)).astype(np.float64)[:20000]) / 2
        a = np.concatenate([v, edge, f.astype(np.float64), ties])
        same(call(lib.t_narrow, a, out=np.float32), a.astype(np.float32))
        same(call(lib.t_widen, f), f.astype(np.float64))


@pytest.mark.parametrize("d", [1, 2, 3, 5, 7, 50, 64, 100, 104, 163, 256, 1023, 1 << 20, (1 << 30) - 1, (1 << 31) - 1])
def test_index_division(lib, d):
    rng = np.random.default_rng(d)
    t = rng.integers(0, 1 << 31, 20000)
    m = np.arange(1, 2000, dtype=np.int64) * d
    t = np.concatenate([t, m, m - 1, m + 1, [0, (1 << 31) - 1]])
    t = t[(t >= 0) & (t < 1 << 31)].astype(np.uint32)
    lib.t_index.restype = ctypes.c_long
    assert lib.t_index(d, t.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(t.size)) == 0
