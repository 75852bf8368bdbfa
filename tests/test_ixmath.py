"""The adjoint's integer transcendentals and its quotients (csrc/lpg_ixmath.cuh)
against CUDA's functions and against long double, at the seams of their tables,
the ends of their ranges, their branch points and between.

Bounds, in units of the result's last place: rounding once is 0.5; beside it
  exp    the cut-off parts of the products, 2^-60 of the result, and of 1/ln 2
         x 2^-64: 0.52 up to x = 32, 0.8 up to 700;
  log1p  2.9 2^-57 from 1 on, 6 2^-63 of at least 2^-5 below: 0.75;
  log2   fixed point with 52 fraction bits, 2^-58 beside the rounding: 0.52;
  n / d  one step from CUDA's correctly rounded quotient, and that for one in
         1e5 at most.
CUDA's exp and log1p are within 1, so they lie at most two steps away."""

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
  if (OP == 0) { ours[i] = ix_exp_neg(T, x[i]); cuda[i] = exp(-x[i]); }
  if (OP == 1) { ours[i] = ix_log1p(T, x[i]); cuda[i] = log1p(x[i]); }
  if (OP == 2) { ours[i] = __longlong_as_double(ix_log2(T, x[i])); cuda[i] = log2(x[i]); }
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
  if (op == 0) k<0><<<g, 256>>>(T, n, d, d + n, d + 2 * n, d + 3 * n);
  if (op == 1) k<1><<<g, 256>>>(T, n, d, d + n, d + 2 * n, d + 3 * n);
  if (op == 2) k<2><<<g, 256>>>(T, n, d, d + n, d + 2 * n, d + 3 * n);
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


def _ulps(got, want):
    """|got - want| in units of want's last place; want in long double."""
    w = want.astype(np.float64)
    return (np.abs(got.astype(np.longdouble) - want) / np.spacing(np.abs(w)).astype(np.longdouble)).astype(np.float64)


def _steps(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64))


def _long_double():
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no long double")


@pytest.mark.gpu
def test_gpu_exp_of_minus_x(device):
    _long_double()
    rng = np.random.default_rng(1)
    seams = np.arange(0, 128 * 1010) * (np.log(2.0) / 128)
    x = np.concatenate([_about(seams[seams < 699.9]), _about([2.0**-7, 0.5, 1.0, 32.0, 2.0**-60, 2.0**-1022]),
                        rng.uniform(0, 700, 200000), rng.uniform(0, 2, 400000), np.exp(rng.uniform(-60, 6.5, 400000)),
                        [0.0, 5e-324, np.nextafter(700.0, 0.0)]])
    x = x[(x >= 0) & (x < 700)]
    ours, cuda = device(0, x)
    err = _ulps(ours, np.exp(-x.astype(np.longdouble)))
    assert err[x <= 32].max() <= 0.52 and err.max() <= 0.8, (err[x <= 32].max(), err.max())
    assert _steps(ours, cuda).max() <= 2


@pytest.mark.gpu
def test_gpu_log1p(device):
    _long_double()
    rng = np.random.default_rng(2)
    m = 1.0 + np.arange(129) / 128.0
    seams = np.concatenate([m * 2.0**e - 1.0 for e in range(0, 60)])
    x = np.concatenate([_about(seams), _about(2.0 ** np.arange(-5, 60)), np.exp(rng.uniform(-3.4, 41.5, 800000)),
                        rng.uniform(2.0**-5, 1.0, 400000), [2.0**-5, np.nextafter(2.0**60, 0.0)]])
    x = x[(x >= 2.0**-5) & (x < 2.0**60)]
    ours, cuda = device(1, x)
    err = _ulps(ours, np.log1p(x.astype(np.longdouble)))
    assert err.max() <= 0.75, err.max()
    assert _steps(ours, cuda).max() <= 2


@pytest.mark.gpu
def test_gpu_log2_in_fixed_point(device):
    _long_double()
    rng = np.random.default_rng(3)
    m = 1.0 + np.arange(129) / 128.0
    big = np.finfo(np.float64).max
    x = np.concatenate([_about(np.concatenate([m * 2.0**e for e in (-1022, -500, -1, 0, 1, 7, 500, 1022)])),
                        2.0 ** rng.uniform(-1022, 1023.99, 400000), rng.uniform(0.5, 4000.0, 400000), [2.0**-1022, big]])
    x = x[(x >= 2.0**-1022) & np.isfinite(x)]
    ours, cuda = device(2, x)
    fixed = ours.view(np.int64)
    want = np.log2(x.astype(np.longdouble)) * np.longdouble(2.0) ** 52
    err = np.abs(fixed.astype(np.longdouble) - want).astype(np.float64)
    assert err.max() <= 0.52, err.max()
    assert np.abs(fixed / 2.0**52 - cuda).max() <= 2.0**-42  # CUDA's, of up to 1024


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
