"""FixedSum itself, in a kernel of this test's own: a sum it calls valid has no
infinite or NaN term, whatever the other factor (zero and tiny weights among
them), takes a large number's product with a zero for the zero it is, and lies
within 15 times 2^-57 of the largest term (what cutting each of at most 15 terms
there can lose) of the exact sum, plus the rounding of the result."""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "softmul.cuh"
__global__ void k(const double *a, const double *b, double *out, int *ok, int rows, int n) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  mpaso::FixedSum s;
  for (int j = 0; j < n; ++j) s.add(a[(int64_t)r * n + j], mpaso::FixedFactor(b[(int64_t)r * n + j]));
  ok[r] = s.valid();
  out[r] = s.valid() ? s.value() : 0.0;
}
extern "C" int run(const double *a, const double *b, double *out, int *ok, int rows, int n) {
  k<<<(rows + 127) / 128, 128>>>(a, b, out, ok, rows, n);
  return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    torch = pytest.importorskip("torch")
    d = tmp_path_factory.mktemp("fixed_sum")
    (d / "k.cu").write_text(SRC)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(ROOT, "mpas-o-flecsi-2.0_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-o", str(d / "k.so"), str(d / "k.cu")], check=True)
    lib = ctypes.CDLL(str(d / "k.so"))

    def call(a, b):
        rows, n = a.shape
        x, y = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (a, b))
        out = torch.zeros(rows, dtype=torch.float64, device="cuda")
        ok = torch.zeros(rows, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        p = [ctypes.c_void_p(v.data_ptr()) for v in (x, y, out, ok)]
        assert lib.run(*p, rows, n) == 0
        return out.cpu().numpy(), ok.cpu().numpy().astype(bool)

    return call


@pytest.mark.parametrize("weight", [0.0, 5e-324, 2.0 ** -300, 2.0 ** -190, 0.1])
@pytest.mark.parametrize("value", [np.nan, np.copysign(np.nan, -1.0), np.inf, -np.inf])
def test_no_sum_over_what_is_no_number(run, value, weight):
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((64, 10)) * 3000.0, rng.uniform(-0.05, 0.05, (64, 10))
    _, ok = run(a, b)
    assert ok.all()
    for r in range(64):
        a[r, r % 10], b[r, r % 10] = value, weight
    _, ok = run(a, b)
    assert not ok.any()


def _check_errors(a, b, out, ok, rows):
    for r in rows:
        if ok[r]:
            terms = [Fraction(float(x)) * Fraction(float(y)) for x, y in zip(a[r], b[r])]
            exact, big = sum(terms), max(abs(t) for t in terms)
            bar = 15 * big / 2 ** 57 + abs(exact) / 2 ** 53
            assert math.isfinite(out[r]) and abs(Fraction(float(out[r])) - exact) <= bar, r


@pytest.mark.parametrize("n", [1, 10, 15])
@pytest.mark.parametrize("spread", [0, 20, 60])
def test_error_of_valid_sums(run, spread, n):
    rng = np.random.default_rng(4)
    a = np.ldexp(rng.standard_normal((4000, n)), rng.integers(-spread, spread + 1, (4000, n)))
    b = rng.uniform(-1.0, 1.0, (4000, n))
    a[rng.uniform(size=a.shape) < 0.1] = 0.0
    b[rng.uniform(size=b.shape) < 0.1] = 0.0
    out, ok = run(a, b)
    assert np.array_equal(ok, (a * b != 0.0).any(axis=1))  # a sum of zeros alone is left to the caller
    _check_errors(a, b, out, ok, range(0, 4000, 7))


@pytest.mark.parametrize("weight", [0.0, 5e-324, -1e-310])
@pytest.mark.parametrize("exp2", [1, 60, 500, 900, 960, 980, 1000, 1023])
def test_large_number_beside_a_zero_weight(run, exp2, weight):
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((64, 10)) * 3000.0, rng.uniform(-0.05, 0.05, (64, 10))
    for r in range(64):
        a[r, r % 10], b[r, r % 10] = 1.5 * 2.0 ** exp2, weight
    out, ok = run(a, b)
    assert ok.all() or exp2 > 900
    _check_errors(a, b, out, ok, range(64))
