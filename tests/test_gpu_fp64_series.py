"""The FP64 reciprocal powers of bh_fp64.cuh over their range, against the x86
80-bit values.

inv_sqrt64: the residual e = 1 - x y^2 is formed with one rounding of x y (an
absolute error of u in e, half of it in the result), the product and the dropped
(5/16) e^3 are far below u for a seed good to 2^-20, and the last operation rounds
once: at most 1.5 u and a little, u = 2^-53; 2 u allowed.
mass_over_r3: y m, y^2 and their product round once each, the rounding of y^2
enters e (1.5 u more), the last operation rounds once: 5.5 u and a little; 6 u."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53

SOURCE = r"""
#include "bh_fp64.cuh"
__global__ void series_kernel(const double *x, const double *m, double *a, double *b, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) { a[i] = bh::inv_sqrt64(x[i]); b[i] = bh::mass_over_r3(x[i], m[i]); }
}
extern "C" int series(const double *x, const double *m, double *a, double *b, int n) {
  series_kernel<<<(n + 127) / 128, 128>>>(x, m, a, b, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def series(tmp_path_factory):
    from hierarquicos_b200 import build

    d = tmp_path_factory.mktemp("series")
    src, so = d / "series.cu", d / "series.so"
    src.write_text(SOURCE)
    subprocess.run([os.environ.get("NVCC", "nvcc"), *build.NVCC_FLAGS, "-I", build.CSRC, "-shared",
                    str(src), "-o", str(so)], check=True)
    f = ctypes.CDLL(str(so)).series

    def run(x, m):
        t = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x, m)]
        out = [torch.empty_like(t[0]) for _ in range(2)]
        assert f(*[ctypes.c_void_p(v.data_ptr()) for v in t + out], len(x)) == 0
        return [v.cpu().numpy() for v in out]

    return run


def _points(lo, hi, n=400000):
    rng = np.random.default_rng(0)
    x = 10.0 ** rng.uniform(np.log10(lo), np.log10(hi), n)
    near = rng.integers(-3, 4, n // 4)  # within three steps of powers of two
    p = np.ldexp(1.0, rng.integers(int(np.log2(lo)) + 1, int(np.log2(hi)), n // 4))
    p = p + near * np.spacing(p)
    return np.concatenate([x, p, rng.uniform(1.0, 4.0, n)])


def test_inverse_square_root(series):
    x = _points(1e-300, 1e300)
    got, _ = series(x, np.ones_like(x))
    ref = 1.0 / np.sqrt(x.astype(np.longdouble))
    assert (np.abs(got - ref) <= 2 * U * ref).all()


def test_mass_over_r_cubed(series):
    x = _points(1e-190, 1e190)
    m = 10.0 ** np.random.default_rng(1).uniform(-12, 12, len(x))
    _, got = series(x, m)
    r = np.sqrt(x.astype(np.longdouble))
    ref = m / (r * x)
    assert (np.abs(got - ref) <= 6 * U * ref).all()


def test_outside_the_range(series):
    """Zero, subnormal, negative and non-finite arguments, and cubes beyond the
    range of a double, are never taken for a finite force."""
    x = np.array([0.0, 5e-324, 2e-308, -1.0, np.inf, np.nan, 1e-220])
    _, b = series(x, np.ones_like(x))
    assert not np.isfinite(b).any()
    _, b = series(np.array([1e220, 1e300]), np.ones(2))
    assert (b == 0.0).all()
