"""csrc/fp64_seed.cuh, compiled into a kernel of its own: reciprocals and reciprocal square
roots over the whole exponent range against values in extended precision, and against what
CUDA's division and square root give where they take over.

Bound: the seed's defect r is formed with one rounding of 2^-53, which enters halved (square
root) or not at all, the result is rounded once (2^-53) and the series is cut below 2^-63: less
than 2^-52."""

import ctypes
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "fp64_seed.cuh"
__global__ void run_kernel(int op, const double* x, const double* y, double* out, long n) {
  const long i = blockIdx.x * 256L + threadIdx.x;
  if (i >= n) return;
  switch (op) {
    case 0: out[i] = ptn::fast_rsqrt(x[i]); break;
    case 1: out[i] = ptn::fast_recip(x[i]); break;
    case 2: out[i] = ptn::half_of(x[i]); break;
    case 3: out[i] = ptn::inv_norm(x[i], y[i]); break;
    case 4: out[i] = 1.0 / sqrt(x[i]); break;
    default: out[i] = 1.0 / x[i]; break;
  }
}
extern "C" int run(int op, const double* x, const double* y, double* out, long n) {
  run_kernel<<<(unsigned)((n + 255) / 256), 256>>>(op, x, y, out, n);
  return (int)cudaDeviceSynchronize();
}
"""
RSQRT, RECIP, HALF, NORM, CUDA_RSQRT, CUDA_RECIP = range(6)


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    import torch
    from pytenet_gb300 import build
    d = tmp_path_factory.mktemp("seed")
    (d / "seed.cu").write_text(SOURCE)
    subprocess.run([build.nvcc_path(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", build.CSRC, str(d / "seed.cu"), "-o", str(d / "seed.so")], check=True,
                   capture_output=True)
    lib = ctypes.CDLL(str(d / "seed.so"))
    lib.run.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]

    def call(op, x, y=None):
        dx = torch.tensor(x, dtype=torch.float64, device="cuda")
        dy = dx if y is None else torch.tensor(y, dtype=torch.float64, device="cuda")
        out = torch.empty_like(dx)
        torch.cuda.synchronize()
        assert lib.run(op, dx.data_ptr(), dy.data_ptr(), out.data_ptr(), len(x)) == 0
        return out.cpu().numpy()

    return call


def samples(lo, hi):
    """Positive numbers of every binary exponent lo .. hi: random, and the ends of each binade."""
    rng = np.random.default_rng(0)
    e = np.arange(lo, hi + 1)
    m = np.concatenate([1 + rng.uniform(0, 1, (64, len(e))), np.ones((1, len(e))),
                        np.full((1, len(e)), 2 - 2.0 ** -52), np.full((1, len(e)), 1 + 2.0 ** -52),
                        np.full((1, len(e)), 1 + 2.0 ** -23 - 2.0 ** -52)])
    return np.ldexp(m, e[None, :]).reshape(-1)


def test_rsqrt_over_the_exponent_range(run):
    x = samples(-1022, 1023)
    ref = 1 / np.sqrt(x.astype(np.longdouble))
    assert float(np.abs(run(RSQRT, x) / ref - 1).max()) < 2.0 ** -52


def test_recip_over_the_exponent_range(run):
    x = samples(-1022, 1021)
    ref = 1 / x.astype(np.longdouble)
    assert float(np.abs(run(RECIP, x) / ref - 1).max()) < 2.0 ** -52


@pytest.mark.parametrize("op,cuda", [(RSQRT, CUDA_RSQRT), (RECIP, CUDA_RECIP)])
def test_ends_of_the_range_are_cudas(run, op, cuda):
    """Zeros, subnormals, infinities, NaN and negative numbers; the recip's last exponents."""
    x = np.concatenate([[0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, -3.5e-200, 5e-324, 2.0 ** -1030,
                         2.2250738585072009e-308], samples(-1074, -1023)])
    if op == RECIP:
        x = np.concatenate([x, samples(-1022, -1022), samples(1018, 1023)])
    a, b = run(op, x), run(cuda, x)
    assert np.array_equal(a, b, equal_nan=True) and np.array_equal(np.signbit(a), np.signbit(b))


def test_half_and_inverse_norm(run):
    x = samples(-900, 1000)
    assert np.array_equal(run(HALF, x), x / 2)
    rng = np.random.default_rng(1)
    t = np.concatenate([rng.uniform(-1, 1, 20000), [0.0, 1.0, -1.0, 1e-12, 1e-200]])
    y = np.ones_like(t)   # cosine of a rotation
    ref = 1 / np.sqrt(t.astype(np.longdouble) ** 2 + 1)
    assert float(np.abs(run(NORM, t, y) / ref - 1).max()) < 2.0 ** -51   # x^2 + y^2 is rounded too
    ph = rng.uniform(0, 2 * np.pi, 20000)   # a phase known to FP32 accuracy
    x, y = np.cos(ph).astype(np.float32).astype(float), np.sin(ph).astype(np.float32).astype(float)
    ref = 1 / np.sqrt(x.astype(np.longdouble) ** 2 + y.astype(np.longdouble) ** 2)
    assert float(np.abs(run(NORM, x, y) / ref - 1).max()) < 2.0 ** -51
