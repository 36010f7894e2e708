"""The step's comparisons, minima and maxima on bit patterns against the FP64 operations they
stand for, over ordinary and limiting values (infinities, zeros, subnormal numbers and the
positive quiet NaN that arithmetic gives on the GPU).
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "uclales_salsa_gb300", "csrc")
# name, bit form, FP64 form, whether the second argument is a positive constant / limit, first may be negative
FORMS = [("num_ge", "num_ge(a, b) ? 1. : 0.", "a >= b ? 1. : 0.", True),
         ("num_gt", "num_gt(a, b) ? 1. : 0.", "a > b ? 1. : 0.", True),
         ("num_lt", "num_lt(a, b) ? 1. : 0.", "a < b ? 1. : 0.", True),
         ("min_pos", "min_pos(a, b)", "fmin(a, b)", True),
         ("max_pos", "max_pos(b, a)", "fmax(b, a)", True),
         ("pos_part", "pos_part(a)", "fmax(0., a)", True),
         ("limit_pos", "limit_pos(a, b)", "fmin(fmax(a, -b), b)", False)]
SOURCE = """
#include "salsa_kernel_impl.cuh"
using namespace salsa;
__global__ void ev(int f, const double *x, const double *y, double *o, double *r, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i], b = y[i];
  switch (f) {
%s
  }
}
extern "C" int eval(int f, const double *x, const double *y, double *o, double *r, int n) {
  ev<<<(n + 255) / 256, 256>>>(f, x, y, o, r, n);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
""" % "\n".join(f"    case {i}: o[i] = {b}; r[i] = {p}; break;" for i, (_, b, p, _) in enumerate(FORMS))
ANY = [0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 1e-300, 1e300, -1e300, 1e-6, 1.0 + 2.0 ** -52, 3.5, -3.5]
POSITIVE = [1e-300, 1e-23, 1e-6, 1.0, 3.5, 1e300]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("bits")
    src, so = d / "ev.cu", d / "ev.so"
    src.write_text(SOURCE)
    cc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([cc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    torch.cuda.init()
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("f", range(len(FORMS)), ids=[n for n, *_ in FORMS])
def test_bit_forms_equal_the_fp64_operations(lib, f):
    second = POSITIVE if FORMS[f][3] else POSITIVE + [0.0, np.inf, np.nan]
    x, y = (a.ravel().copy() for a in np.meshgrid(np.array(ANY), np.array(second)))
    tx, ty = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    o, r = torch.empty_like(tx), torch.empty_like(tx)
    torch.cuda.synchronize()
    assert lib.eval(f, *[ctypes.c_void_p(t.data_ptr()) for t in (tx, ty, o, r)], x.size) == 0
    got, ref = o.cpu().numpy(), r.cpu().numpy()
    bad = ~((got == ref) | (np.isnan(got) & np.isnan(ref)))
    assert not bad.any(), list(zip(x[bad], y[bad], got[bad], ref[bad]))[:5]
