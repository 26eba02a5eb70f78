"""The leaf offsets of the sweep (leaf_narrow, leaf_wide in csrc/dev_common.cuh)
as compiled, in a kernel of their own, against exact integers: the last number
of the longest segment, the largest divisors, remainders 0 and m - 1, and xp's
high word left out."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "dev_common.cuh"
using namespace pcg;
__global__ void k_offsets(int wide, int n, const uint64_t* xlo, const uint64_t* low, const uint32_t* m, uint32_t* out)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = wide ? leaf_wide(xlo[i], low[i], m[i]) : leaf_narrow(xlo[i], low[i], m[i]);
}
extern "C" int span_max() { return (int) LEAF_SPAN; }
extern "C" int offsets(int wide, int n, const uint64_t* xlo, const uint64_t* low, const uint32_t* m, uint32_t* out)
{
  char* d = nullptr;
  const size_t n8 = (size_t) n * 8, n4 = (size_t) n * 4;
  if (cudaMalloc(&d, 2 * n8 + 2 * n4) != cudaSuccess) return 1;
  cudaMemcpy(d, xlo, n8, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n8, low, n8, cudaMemcpyHostToDevice);
  cudaMemcpy(d + 2 * n8, m, n4, cudaMemcpyHostToDevice);
  k_offsets<<<(n + 255) / 256, 256>>>(wide, n, (const uint64_t*) d, (const uint64_t*) (d + n8),
                                      (const uint32_t*) (d + 2 * n8), (uint32_t*) (d + 2 * n8 + n4));
  const cudaError_t e = cudaMemcpy(out, d + 2 * n8 + n4, n4, cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e != cudaSuccess;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from primecount_gb300 import build
    d = tmp_path_factory.mktemp("leaf")
    src, so = str(d / "leaf.cu"), str(d / "leaf.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build._nvcc()] + build.ARCH + build.NVCC_FLAGS + ["-shared", src, "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("wide", [0, 1])
def test_offsets_are_exact(lib, wide):
    span = 1 << 23 if wide else lib.span_max()
    assert wide or span == 1 << 21
    mtop = (1 << 32) - 1 if wide else (1 << 30) - 1
    rng = np.random.default_rng(11 + wide)
    n = 1 << 20
    m = np.exp(rng.uniform(0, np.log(mtop), n)).astype(np.uint64)
    m = np.clip(m, 1, mtop)
    m[::4] = mtop - rng.integers(0, 3, m[::4].size).astype(np.uint64)
    d = np.exp(rng.uniform(0, np.log(span), n)).astype(np.uint64)
    d[::3] = span - 1 - rng.integers(0, 3, d[::3].size).astype(np.uint64)
    d[1::7] = rng.integers(0, 3, d[1::7].size).astype(np.uint64)
    d = np.minimum(d, span - 1)
    t = (rng.random(n) * m.astype(np.float64)).astype(np.uint64)
    t[::5] = 0
    t[1::5] = m[1::5] - np.uint64(1)
    t = np.minimum(t, m - np.uint64(1))
    low = rng.integers(0, 10 ** 16, n).astype(np.uint64) // np.uint64(240) * np.uint64(240)
    low[:1000] = 0
    xlo = (low + d) * m + t                      # the low word of xp, modulo 2^64
    m32 = m.astype(np.uint32)
    out = np.zeros(n, dtype=np.uint32)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert lib.offsets(wide, n, ptr(xlo), ptr(low), ptr(m32), ptr(out)) == 0
    bad = np.nonzero(out != d)[0]
    assert bad.size == 0, [(int(m[i]), int(d[i]), int(t[i]), int(out[i])) for i in bad[:5]]
