"""The adjoint's quotients (csrc/lpg_ixmath.cuh) against CUDA's: one step from
CUDA's correctly rounded quotient, and that for one in 1e5 at most."""


import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "laser_polio_gb300" / "csrc"

SOURCE = r"""
#include "lpg_ixmath.cuh"
template <int OP>
__global__ void k(const IxTables* T, int n, const double* x, const double* y, double* ours, double* cuda) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  if (OP == 3) { ours[i] = IxDivisor(y[i]).of(x[i]); cuda[i] = x[i] / y[i]; }
}
extern "C" int run(int op, int n, const double* x, const double* y, double* ours, double* cuda) {
  double* d = nullptr;
  IxTables* T = nullptr;
  const size_t b = sizeof(double) * n;
  if (cudaMalloc((void**)&d, 4 * b) || cudaMalloc((void**)&T, sizeof(IxTables))) return 1;
  cudaMemcpy(T, ix_tables(), sizeof(IxTables), cudaMemcpyHostToDevice);
  cudaMemcpy(d, x, b, cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, y, b, cudaMemcpyHostToDevice);
  const int g = (n + 255) / 256;
  if (op == 3) k<3><<<g, 256>>>(T, n, d, d + n, d + 2 * n, d + 3 * n);
  cudaMemcpy(ours, d + 2 * n, b, cudaMemcpyDeviceToHost);
  cudaMemcpy(cuda, d + 3 * n, b, cudaMemcpyDeviceToHost);
  const int rc = cudaDeviceSynchronize() != cudaSuccess || cudaGetLastError() != cudaSuccess;
  cudaFree(d);
  cudaFree(T);
  return rc;
}
"""


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    from laser_polio_gb300.build import ARCH
    from laser_polio_gb300.build import FLAGS
    from laser_polio_gb300.build import nvcc

    d = tmp_path_factory.mktemp("ixmath")
    (d / "t.cu").write_text(SOURCE)
    subprocess.run([nvcc(), ARCH, *FLAGS, "-shared", f"-I{CSRC}", str(d / "t.cu"), "-o", str(d / "t.so")], check=True)
    lib = C.CDLL(str(d / "t.so"))

    def call(op, x, y=None):
        x = np.ascontiguousarray(x, np.float64)
        y = np.ones_like(x) if y is None else np.ascontiguousarray(y, np.float64)
        ours, cuda = np.empty_like(x), np.empty_like(x)
        p = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in (x, y, ours, cuda)]
        assert lib.run(op, len(x), *p) == 0
        return ours, cuda

    return call


def _about(points, steps=6):
    """The points and their neighbours a few steps away."""
    out = [np.asarray(points, np.float64)]
    lo = hi = out[0]
    for _ in range(steps):
        lo, hi = np.nextafter(lo, -np.inf), np.nextafter(hi, np.inf)
        out += [lo, hi]
    return np.concatenate(out)


def _steps(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64))


@pytest.mark.gpu
def test_gpu_quotients(device):
    rng = np.random.default_rng(4)
    n = 1000000
    d = np.concatenate([np.exp(rng.uniform(0, 346, n)), rng.uniform(1, 2, n), rng.integers(1, 1 << 30, n).astype(np.float64)])
    x = np.concatenate([np.exp(rng.uniform(-345, 345, n)), rng.uniform(-2, 2, n), rng.integers(-(1 << 30), 1 << 30, n) * 1.0])
    ours, cuda = device(3, x, d)
    s = _steps(ours, cuda)
    assert s.max() <= 1 and (s != 0).mean() <= 1e-5, (s.max(), (s != 0).mean())
    # what goes to the general division: the same bits
    big = np.finfo(np.float64).max
    edge = np.array([0.0, -0.0, 5e-324, 1e-310, 2.0**-501, 2.0**500, 1e300, big, np.inf, -np.inf, np.nan, 1.0, -1.0, 0.5, -3.0])
    d, x = (a.ravel() for a in np.meshgrid(edge, np.concatenate([edge, _about([1.0, 2.0**500, 2.0**-500])])))
    ours, cuda = device(3, x, d)
    same = (ours == cuda) | (np.isnan(ours) & np.isnan(cuda))
    assert same.all(), (x[~same][:5], d[~same][:5])
