"""The key sort when a block does not wait for the blocks before it (GPU): the
sort's source built with no waiting at all, so that a block which does not find
its predecessors' totals at once counts their keys itself."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r'''
#include "rk_prims.cu"
extern "C" int sort_keys(uint64_t* keys, uint64_t* tmp, long n, int lo, int hi) {
  void* temp = nullptr;
  if (cudaMalloc(&temp, rk::sort_temp_bytes(n)) != cudaSuccess) return -1;
  rk::radix_sort_u64(keys, tmp, n, lo, hi, temp, 0);
  const cudaError_t e = cudaDeviceSynchronize();
  cudaFree(temp);
  return (int)e;
}
'''


@pytest.fixture(scope="module")
def impatient(gpu_lib, tmp_path_factory):
    from rockable_gb300 import build_ext
    d = tmp_path_factory.mktemp("sort")
    src, so = d / "sort.cu", d / "sort.so"
    src.write_text(SRC)
    subprocess.check_call([build_ext.nvcc(), build_ext.GENCODE, "-O3", "-std=c++17", "-DRK_SORT_SPINS=0", "-shared",
                           "-Xcompiler", "-fPIC", "-I", build_ext.CSRC, str(src), "-o", str(so)])
    L = ctypes.CDLL(str(so))
    L.sort_keys.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_int, ctypes.c_int]
    return L


@pytest.mark.parametrize("n,lo,hi", [(4096, 0, 64), (4097, 0, 64), (300001, 0, 64), (200000, 27, 51), (1000003, 22, 59)])
def test_the_sort_does_not_depend_on_the_wait(n, lo, hi, impatient):
    import torch
    a = np.random.default_rng(n).integers(0, 2 ** 63 - 1, n, dtype=np.int64)
    t, tmp = torch.from_numpy(a.copy()).cuda(), torch.empty(n, dtype=torch.int64, device="cuda")
    assert impatient.sort_keys(t.data_ptr(), tmp.data_ptr(), n, lo, hi) == 0
    u = a.view(np.uint64)
    digits = (u >> np.uint64(lo)) & np.uint64((1 << (hi - lo)) - 1)
    assert np.array_equal(t.cpu().numpy().view(np.uint64), u[np.argsort(digits, kind="stable")])
