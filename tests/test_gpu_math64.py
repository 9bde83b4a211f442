"""The FP64 functions with few FP64 instructions (lacmo_math64.cuh, lacmo_ff.cuh)
against CUDA's own, value by value over their ranges.

Bounds.  Reciprocal, quotient: within 0.51 of a last place, CUDA's are correctly
rounded: one last place apart at most.  Square root: half the rounding of x z is
left, 0.8 of a last place: one apart.  Cube root (two roundings in the residual),
exp and log (some 2.5 roundings of 2^-53 beside the last): CUDA's are within one
last place: 2^-50 relative in all."""
import ctypes
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SOURCE = """
#include "lacmo_math64.cuh"
using namespace lacmo;
__global__ void k_eval(int f, long long n, const double* x, const double* y, double* a, double* b) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
       k += (long long)gridDim.x * blockDim.x) {
    const double u = x[k], v = y[k];
    switch (f) {
      case 0: a[k] = rcp64(u); b[k] = 1.0 / u; break;
      case 1: a[k] = div64(u, v); b[k] = u / v; break;
      case 2: a[k] = sqrt64(u); b[k] = sqrt(u); break;
      case 3: a[k] = icbrt64(u); b[k] = rcbrt(u); break;
      case 4: a[k] = exp64(u); b[k] = exp(u); break;
      case 5: a[k] = log64(u); b[k] = log(u); break;
      default: {
        const ff p = ff_quick((float)u, (float)(u - (double)(float)u));
        a[k] = ff2d_int(p); b[k] = ff2d(p);
      }
    }
  }
}
extern "C" int eval(int f, long long n, const double* x, const double* y, double* a, double* b) {
  k_eval<<<1024, 128>>>(f, n, x, y, a, b);
  return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def ev(tmp_path_factory):
    from lacmopy_gb300 import build
    d = tmp_path_factory.mktemp("math64")
    (d / "eval.cu").write_text(SOURCE)
    out = str(d / "eval.so")
    subprocess.run([build._nvcc(), "-shared", "-o", out, str(d / "eval.cu")] + build.COMMON,
                   check=True)
    lib = ctypes.CDLL(out)

    def run(f, x, y=None):
        x = torch.as_tensor(x, dtype=torch.float64, device="cuda")
        y = x if y is None else torch.as_tensor(y, dtype=torch.float64, device="cuda")
        a, b = torch.empty_like(x), torch.empty_like(x)
        torch.cuda.synchronize()
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in (x, y, a, b)]
        assert lib.eval(f, ctypes.c_longlong(x.numel()), *ptr) == 0
        return a.cpu().numpy(), b.cpu().numpy()
    return run


N = 2_000_000


def _wide(seed, lo, hi, sign=False):
    """Magnitudes spread over 2^lo to 2^hi, with powers of two and their neighbours."""
    rng = np.random.default_rng(seed)
    x = 2.0 ** rng.uniform(lo, hi, N)
    p = 2.0 ** np.arange(lo + 1, hi)
    edge = np.concatenate([p, np.nextafter(p, 0), np.nextafter(p, np.inf)])
    x[:edge.size] = edge
    return x * rng.choice([-1.0, 1.0], N) if sign else x


def _places(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64)).max()


def test_reciprocal_and_quotient(ev):
    assert _places(*ev(0, _wide(1, -120, 120, sign=True))) <= 1
    assert _places(*ev(1, _wide(2, -100, 100, sign=True), _wide(3, -100, 100, sign=True))) <= 1


def test_outside_the_range(ev):
    """Infinities, NaN, zeros and numbers beyond FP32: as the library."""
    v = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, 5e-324, 1e-300, -1e-60, 1e-39, 1.0,
                  -3.0, 1e37, 1e39, -1e60, 1e200, 1.7e308])
    x, y = (t.ravel() for t in np.meshgrid(v, v))
    a, b = ev(1, x, y)
    nan = np.isnan(b)
    assert np.array_equal(np.isnan(a), nan)
    ulp = np.abs(a[~nan].view(np.int64) - b[~nan].view(np.int64))
    assert np.array_equal(np.signbit(a[~nan]), np.signbit(b[~nan])) and ulp.max() <= 1
    a, b = ev(2, v)
    np.testing.assert_array_equal(a[[0, 1, 2, 3, 4, 5, 6, 7, 8, 13, 14, 15, 16]],
                                  b[[0, 1, 2, 3, 4, 5, 6, 7, 8, 13, 14, 15, 16]])


def test_roots(ev):
    assert _places(*ev(2, _wide(4, -120, 120))) <= 1
    a, b = ev(3, _wide(5, -100, 100))
    assert np.abs(a / b - 1).max() <= 2.0 ** -50


@pytest.mark.parametrize("span", [1e-6, 0.5, 3.0, 50.0, 700.0])
def test_exp(ev, span):
    x = np.random.default_rng(6).uniform(-span, span, N)
    half = (np.arange(-800, 800) + 0.5) * np.log(2.0)
    x[:half.size] = np.clip(half, -span, span)
    x[-4:] = (0.0, -0.0, 800.0, -800.0)
    a, b = ev(4, x)
    assert np.array_equal(a[-4:], b[-4:])
    assert np.abs(a[:-4] / b[:-4] - 1).max() <= 2.0 ** -50


@pytest.mark.parametrize("lo,hi", [(-1000, 1000), (-3, 3), (-1e-3, 1e-3)])
def test_log(ev, lo, hi):
    x = 2.0 ** np.random.default_rng(7).uniform(lo, hi, N)
    x[-5:] = (1.0, 0.0, -1.0, np.inf, 5e-324)
    a, b = ev(5, x)
    np.testing.assert_array_equal(a[-5:], b[-5:])
    a, b = a[:-5], b[:-5]
    one = b == 0.0
    assert np.array_equal(a[one], b[one])
    assert np.abs(a[~one] / b[~one] - 1).max() <= 2.0 ** -50


def test_two_floats_to_double(ev):
    """With and without an FP64 instruction: the same bits."""
    a, b = ev(6, _wide(8, -140, 120, sign=True))
    assert np.array_equal(a.view(np.int64), b.view(np.int64))
    x = _wide(9, -20, 20, sign=True)
    x[:1000] = np.float32(x[:1000])   # no low part
    a, b = ev(6, x)
    assert np.array_equal(a.view(np.int64), b.view(np.int64))
