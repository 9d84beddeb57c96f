"""fast_rsqrt and fast_rcp of rot.cuh over the range that they are stated for, against long double.

Bounds, relative: the second Newton step starts from at most 2^-40, so what is left are its own
roundings: of x y (2^-54 after the step's half) and of the result (2^-53) for the root, of the result alone
for the reciprocal, whose residual is exact."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

KERNEL = r"""
#include "rot.cuh"
__global__ void k(const double* x, double* r, double* q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    r[i] = sqg::fast_rsqrt(x[i]);
    q[i] = sqg::fast_rcp(x[i]);
  }
}
extern "C" int run(const double* x, double* r, double* q, int n) {
  k<<<(n + 255) / 256, 256>>>(x, r, q, n);
  return (int)cudaDeviceSynchronize();
}
"""


def test_newton_steps_to_a_rounding(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                        "sequential-quantum-gate-decomposer_gb300", "csrc")
    src, so = tmp_path / "newton.cu", tmp_path / "newton.so"
    src.write_text(KERNEL)
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                           "-fPIC", "-I", csrc, "-o", str(so), str(src)])
    lib = ctypes.CDLL(str(so))
    rng = np.random.default_rng(0)
    powers = np.ldexp(1.0, np.arange(-120, 121))
    x = np.concatenate([powers, np.nextafter(powers, 0), np.nextafter(powers, np.inf),
                        np.ldexp(rng.uniform(1, 2, 200000), rng.integers(-120, 120, 200000)), 1.0 + rng.random(100000)])
    d = torch.from_numpy(x).cuda()
    r, q = torch.empty_like(d), torch.empty_like(d)
    torch.cuda.synchronize()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    assert lib.run(ptr(d), ptr(r), ptr(q), len(x)) == 0
    exact = x.astype(np.longdouble)
    root = np.abs(r.cpu().numpy() * np.sqrt(exact) - 1)
    inverse = np.abs(q.cpu().numpy() * exact - 1)
    assert np.max(root) <= 1.52 * 2.0 ** -53
    assert np.max(inverse) <= 1.01 * 2.0 ** -53
