"""The FP64 functions of csrc/salsa_math.cuh against 64-bit-mantissa (or wider) references.

Each function is evaluated on a GB300 for seeded arguments over its range, for arguments
next to the powers of two, of four and of eight (the ends of the seeds' binades), and for
the arguments that leave the fast path.  The bound is the error of the last rounding (half
an ulp) plus what the method adds: 2^-30 ulp for quotients and square roots (a seed error e
leaves e^2), 0.01 ulp for the cube root, 0.03 for log (the series' last term at its ends),
0.13 for exp (log2(e) to 64 bits times |x| up to 708) and 0.75 for pow (the logarithm's
2^-63 times |y ln x| up to 708).  np.longdouble has 64 or 113 bits; references with 64 bits
add 2^-11 ulp.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "uclales_salsa_gb300", "csrc")
NAMES = ["ddiv", "drcp", "dsqrt", "dcbrt", "dexp", "dlog", "dpow", "divc"]
SOURCE = """
#include "salsa_math.cuh"
using namespace salsa;
__global__ void ev(int f, const double *x, const double *y, double *o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = x[i], b = y[i];
  double r = 0.;
  switch (f) {
    case 0: r = ddiv(a, b); break;
    case 1: r = drcp(a); break;
    case 2: r = dsqrt(a); break;
    case 3: r = dcbrt(a); break;
    case 4: r = dexp(a); break;
    case 5: r = dlog(a); break;
    case 6: r = dpow(a, b); break;
    case 7: r = divc(a, 0.5235988); break;
  }
  o[i] = r;
}
extern "C" int eval(int f, const double *x, const double *y, double *o, int n) {
  ev<<<(n + 255) / 256, 256>>>(f, x, y, o, n);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
"""


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


def ev(lib, name, x, y=None):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.ones_like(x) if y is None else np.ascontiguousarray(y, dtype=np.float64)
    tx, ty = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    o = torch.empty_like(tx)
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in (tx, ty, o)]
    assert lib.eval(NAMES.index(name), *p, x.size) == 0
    return o.cpu().numpy()


def reference(name, x, y):
    L = np.longdouble
    x, y = x.astype(L), y.astype(L)
    return {"ddiv": lambda: x / y, "drcp": lambda: 1 / x, "dsqrt": lambda: np.sqrt(x), "dcbrt": lambda: np.cbrt(x),
            "dexp": lambda: np.exp(x), "dlog": lambda: np.log(x), "dpow": lambda: np.power(x, y),
            "divc": lambda: x / L(0.5235988)}[name]()


N = 200000
BOUND = {"ddiv": 0.501, "drcp": 0.501, "dsqrt": 0.501, "dcbrt": 0.511, "dexp": 0.631, "dlog": 0.531, "dpow": 1.251,
         "divc": 0.501}


def arguments(name, where, rng):
    logu = lambda a, b: np.exp(rng.uniform(np.log(a), np.log(b), N))
    sign = np.where(rng.random(N) < 0.5, -1.0, 1.0)
    y = np.ones(N)
    near = np.ldexp(1.0 + rng.integers(-2000, 2001, N) * 2.0 ** -52, rng.integers(-90, 91, N))   # next to powers of two
    if name in ("ddiv", "drcp", "divc"):
        if where == "range":
            return logu(1e-140, 1e140) * sign, logu(1e-140, 1e140) * sign[::-1]
        return near * sign, near[::-1].copy()
    if name in ("dsqrt", "dcbrt"):
        return (logu(1e-140, 1e140) if where == "range" else near), y
    if name == "dexp":
        return (rng.uniform(-708, 708, N) if where == "range" else rng.integers(-40, 41, N) * np.log(2.0) / 128 *
                (1 + rng.integers(-3, 4, N) * 2.0 ** -50)), y
    if name == "dlog":
        return (logu(1e-300, 1e300) if where == "range" else 1.0 + sign * logu(1e-15, 0.5)), y
    if where == "range":
        x = logu(1e-12, 1e12)
        return x, rng.uniform(-8, 8, N)
    return 1.0 + sign * logu(1e-9, 0.4), rng.uniform(-500, 500, N)


@pytest.mark.parametrize("where", ["range", "edges"])
@pytest.mark.parametrize("name", NAMES)
def test_error_in_ulps(lib, name, where):
    rng = np.random.default_rng(NAMES.index(name) * 2 + (where == "edges"))
    x, y = arguments(name, where, rng)
    got, ref = ev(lib, name, x, y), reference(name, x, y)
    assert np.isfinite(got).all()
    ulp = np.spacing(np.abs(ref.astype(np.float64)))
    # the spacing above a power of two is twice the one below it
    err = np.abs(got.astype(np.longdouble) - ref) / ulp
    assert float(err.max()) <= BOUND[name], float(err.max())


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, -1e-310, 5e-324, 1e308, -1e308, 1.0, -1.0, 2.5e-308, 1e-200,
                    -1e-200, 1e200, 745.0, -745.0, -746.0, 710.0])


@pytest.mark.parametrize("name", NAMES)
def test_arguments_outside_the_fast_range(lib, name):
    x, y = (a.ravel() for a in np.meshgrid(SPECIAL, SPECIAL))
    got = ev(lib, name, x, y)
    with np.errstate(all="ignore"):
        ref = {"ddiv": lambda: x / y, "drcp": lambda: 1.0 / x, "dsqrt": lambda: np.sqrt(x), "dcbrt": lambda: np.cbrt(x),
               "dexp": lambda: np.exp(x), "dlog": lambda: np.log(x), "dpow": lambda: np.power(x, y),
               "divc": lambda: x / 0.5235988}[name]()
    same = (got == ref) | (np.isnan(got) & np.isnan(ref))
    # results of the functions within two ulps (or two subnormal steps) of numpy's
    with np.errstate(all="ignore"):
        near = np.isfinite(ref) & (np.abs(got - ref) <= 4.5e-16 * np.abs(ref) + 1e-323)
    assert (same | near).all(), [(a, b, g, r) for a, b, g, r, s in zip(x, y, got, ref, same | near) if not s][:5]
