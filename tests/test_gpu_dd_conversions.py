"""dd_from_double and dd_to_double (sgba_dd.cuh) form their results from the
mantissas: every bit must be that of the IEEE conversions (numpy's float32 and
float64 arithmetic, round to nearest even).  A small library built from the
header runs them over the edges: exponents inside, at and outside the integer
path's range, ties and near-ties of the 24-bit rounding, carries into the next
binade, zeros of both signs, denormals and infinities."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cuda_runtime.h>
#include "sgba_dd.cuh"
__global__ void k_from(const double* x, float2* o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { const dd v = dd_from_double(x[i]); o[i] = make_float2(v.hi, v.lo); }
}
__global__ void k_to(const float2* x, double* o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) o[i] = dd_to_double(dd_make(x[i].x, x[i].y));
}
extern "C" int convert(const double* x, float2* s, double* back, int n) {
  double *dx, *db; float2* ds;
  if (cudaMalloc(&dx, 8 * n) || cudaMalloc(&db, 8 * n) || cudaMalloc(&ds, 8 * n)) return 1;
  cudaMemcpy(dx, x, 8 * n, cudaMemcpyHostToDevice);
  k_from<<<(n + 127) / 128, 128>>>(dx, ds, n);
  cudaMemcpy(s, ds, 8 * n, cudaMemcpyDeviceToHost);
  k_to<<<(n + 127) / 128, 128>>>(ds, db, n);
  cudaMemcpy(back, db, 8 * n, cudaMemcpyDeviceToHost);
  cudaFree(dx); cudaFree(db); cudaFree(ds);
  return static_cast<int>(cudaGetLastError());
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("dd")
    (d / "conv.cu").write_text(SRC)
    so = str(d / "conv.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-I", os.path.join(ROOT, "sophus-rs_gb300", "csrc"), str(d / "conv.cu"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("lo_exp,hi_exp", [(-5, 5), (-80, -70), (120, 130), (-160, -120), (-1074, -1000), (1000, 1023)])
def test_conversions_match_ieee(lib, lo_exp, hi_exp):
    rng = np.random.default_rng(hi_exp + 2000)
    n = 4096
    frac = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    frac[0::4] &= ~np.uint64(0x1FFFFFFF)                                        # 24 bits
    frac[1::8] = (frac[1::8] & ~np.uint64(0x1FFFFFFF)) | np.uint64(0x10000000)  # ties
    frac[2::8] = (frac[2::8] & ~np.uint64(0x1FFFFFFF)) | np.uint64(0x10000001)
    frac[3::8] = np.uint64((1 << 52) - 1)                                       # carries
    x = np.ldexp(1.0 + frac.astype(np.float64) * 2.0 ** -52, rng.integers(lo_exp, hi_exp + 1, n))
    x *= rng.choice([-1.0, 1.0], n)
    x[:4] = [0.0, -0.0, np.inf, -np.inf]
    with np.errstate(all="ignore"):
        hi = x.astype(np.float32)
        lo = (x - hi.astype(np.float64)).astype(np.float32)
        back = hi.astype(np.float64) + lo.astype(np.float64)
    s, b = np.empty((n, 2), np.float32), np.empty(n)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert lib.convert(ptr(x), ptr(s), ptr(b), n) == 0
    nan = np.isnan(lo)
    assert np.array_equal(s[:, 0].view(np.uint32), hi.view(np.uint32))
    assert np.array_equal(s[~nan, 1].view(np.uint32), lo[~nan].view(np.uint32)) and np.isnan(s[nan, 1]).all()
    nan = np.isnan(back)
    assert np.array_equal(b[~nan].view(np.uint64), back[~nan].view(np.uint64)) and np.isnan(b[nan]).all()
