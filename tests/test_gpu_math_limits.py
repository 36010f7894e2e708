"""Zero, subnormal, infinite, NaN and extreme arguments of the quotients of
csrc/salsa_math.cuh that have an operand at hand: ddiv_r (the reciprocal of the denominator)
and divc (a compile-time constant).  The results are those of the plain division: equal, NaN
where it is NaN, or within two ulps (two subnormal steps).  The constants have 1/c with a low
part of either sign.
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
CONSTANTS = [1000.0, 18.016e-3, 917.0, 400.0, 0.5235988, 296.16, 1.3807e-23, 6.626070040e-34, 3.0, 6.0221e23]
SOURCE = """
#include "salsa_math.cuh"
using namespace salsa;
__global__ void ev(int f, const double *x, const double *y, double *o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i], b = y[i];
  double r = 0.;
  switch (f) {
    case 0: r = ddiv_r(a, b, drcp(b)); break;
%s
  }
  o[i] = r;
}
extern "C" int eval(int f, const double *x, const double *y, double *o, int n) {
  ev<<<(n + 255) / 256, 256>>>(f, x, y, o, n);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
""" % "\n".join(f"    case {i + 1}: r = divc(a, {c!r}); break;" for i, c in enumerate(CONSTANTS))
SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, -1e-310, 5e-324, 1e308, -1e308, 1.0, -1.0, 2.5e-308, 1e-200,
                    -1e-200, 1e200, 1e270, -1e270, 3.0, 1e-150, 1e150])


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    src, so = d / "ev.cu", d / "ev.so"
    src.write_text(SOURCE)
    cc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([cc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", CSRC, str(src), "-o", str(so)], check=True)
    torch.cuda.init()
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("f", range(len(CONSTANTS) + 1))
def test_quotients_of_special_arguments(lib, f):
    x, y = (a.ravel().copy() for a in np.meshgrid(SPECIAL, SPECIAL if f == 0 else np.array([CONSTANTS[f - 1]])))
    tx, ty = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    o = torch.empty_like(tx)
    torch.cuda.synchronize()
    assert lib.eval(f, *[ctypes.c_void_p(t.data_ptr()) for t in (tx, ty, o)], x.size) == 0
    got = o.cpu().numpy()
    with np.errstate(all="ignore"):
        ref = x / y
        same = ((got == ref) & (np.signbit(got) == np.signbit(ref))) | (np.isnan(got) & np.isnan(ref))
        near = np.isfinite(ref) & (np.abs(got - ref) <= 4.5e-16 * np.abs(ref) + 1e-323)
    bad = ~(same | near)
    assert not bad.any(), list(zip(x[bad], y[bad], got[bad], ref[bad]))[:5]
