"""The FP64 operations done on the bits or by a known reciprocal (mcx_exact.h) and the device's short cuts in the
portable exp, log, log10 and pow (mcx_fmath.h), at the edges of what they take: on the host against numpy, on the
GPU against the host."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "mocassin_xray_gb300" / "csrc"

SOURCE = """
#include "mcx_exact.h"
MCX_FM_FN double one(int what, double a, double b) {
  switch (what) {
    case 0: return exactSum(a, b) ? 1. : 0.;
    case 1: return eqDivide(a, b, 1. / b);
    case 2: return mcx_fm_exp(a);
    case 3: return mcx_fm_log(a);
    case 4: return mcx_fm_log10(a);
    default: return mcx_fm_pow(a, b);
  }
}
extern "C" void host(int what, const double* a, const double* b, double* out, long n) {
  for (long i = 0; i < n; ++i) out[i] = one(what, a[i], b[i]);
}
#ifdef __CUDACC__
__global__ void kernel(int what, const double* a, const double* b, double* out, long n) {
  const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (i < n) out[i] = one(what, a[i], b[i]);
}
extern "C" int device(int what, const double* a, const double* b, double* out, long n) {
  double* d = nullptr;
  if (cudaMalloc(&d, 3 * n * sizeof(double)) != cudaSuccess) return 1;
  cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  kernel<<<(unsigned)((n + 255) / 256), 256>>>(what, d, d + n, d + 2 * n, n);
  const cudaError_t e = cudaMemcpy(out, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? 0 : 2;
}
#endif
"""
EXACT, DIVIDE, EXP, LOG, LOG10, POW = range(6)


def _evaluate(fn, what, a, b):
    a, b = (np.ascontiguousarray(np.broadcast_to(x, np.broadcast(a, b).shape), np.float64).ravel() for x in (a, b))
    out = np.empty_like(a)
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, out)]
    assert not fn(what, *p, ctypes.c_long(a.size))
    return a, b, out


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(CSRC), "t.cpp", "-o", "t.so"],
                   cwd=d, check=True)
    f = ctypes.CDLL(str(d / "t.so")).host
    f.restype = None
    return f


def _sums(rng):
    """Pairs of a sum and an FP32 deposit by the gap of their exponents, mantissas odd, even, short and long."""
    gap = np.repeat(np.arange(-60, 61), 400)
    e = rng.integers(-60, 60, gap.size)
    mv = (1 << 23) + rng.integers(0, 1 << 23, gap.size)
    mo = (1 << 52) + rng.integers(0, 1 << 52, gap.size)
    mo = mo >> rng.integers(0, 53, gap.size) << 0
    mo = np.where(rng.random(gap.size) < 0.5, mo, (mo >> 1) << 1)
    shift = 52 - np.floor(np.log2(mo)).astype(int)
    shift = np.clip(shift, 0, 52)
    old = np.ldexp(mo.astype(np.float64), e + gap - 52 + shift)
    v = np.ldexp(mv.astype(np.float64), e - 23)
    special = [0.0, -0.0, 5e-324, 1e-310, 2.2250738585072014e-308, np.inf, np.nan, -1.0, 1.0, 1.7976931348623157e308]
    so, sv = (x.ravel() for x in np.meshgrid(special, np.float32([1e-45, 1e-38, 1.0, 3e38, np.inf, np.nan]).astype(float)))
    return np.concatenate([old, so]), np.concatenate([v, sv])


def _quotients(rng):
    """Quotients over the window of exponents, at its edges and beyond, and of the extreme mantissas."""
    ea, ed = (np.concatenate([rng.integers(-460, 461, 60000), rng.choice([-452, -451, -450, -449, 448, 449, 450, 451], 60000),
                              rng.integers(-1070, 1020, 20000)]) for _ in range(2))
    m = [np.where(rng.random(ea.size) < 0.2, rng.choice([1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52], ea.size),
                  1.0 + rng.random(ea.size)) * rng.choice([-1.0, 1.0], ea.size) for _ in range(2)]
    special = [0.0, -0.0, 1.0, -3.0, 5e-324, 1e308, np.inf, -np.inf, np.nan]
    sa, sd = (x.ravel() for x in np.meshgrid(special, special))
    return np.concatenate([np.ldexp(m[0], ea), sa]), np.concatenate([np.ldexp(m[1], rng.permutation(ed)), sd])


def _arguments(what, rng):
    edge = np.array([672.0, 671.9999, 704.0, 709.782712893384, 709.79, 745.1332191019412, 745.14, 1.0, 0.5, 2.0, 1e-300,
                     2.2250738585072014e-308, 2.225073858507201e-308, 5e-324, 0.0, 1.7976931348623157e308, np.inf, np.nan,
                     10.0, 3.0, 1.5, 1e4])
    edge = np.concatenate([edge, np.nextafter(edge, np.inf), np.nextafter(edge, -np.inf)])
    edge = np.concatenate([edge, -edge])
    if what == POW:
        a, b = (x.ravel() for x in np.meshgrid(edge, edge))
        return np.concatenate([a, 10.0 ** rng.uniform(-300, 300, 50000)]), np.concatenate([b, rng.uniform(-40, 40, 50000)])
    a = np.concatenate([edge, rng.uniform(-750, 750, 50000) if what == EXP else 10.0 ** rng.uniform(-320, 308, 50000)])
    return a, np.zeros_like(a)


def _same(x, y):
    """The same bits, NaN of any sign and payload for NaN."""
    return np.array_equal(np.isnan(x), np.isnan(y)) and np.array_equal(x[~np.isnan(x)].view(np.uint64),
                                                                      y[~np.isnan(y)].view(np.uint64))


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
def test_exact_sum(host):
    """A sum called exact has no rounding error (TwoSum), and those of the binades that count are seen."""
    old, v, got = _evaluate(host, EXACT, *_sums(np.random.default_rng(1)))
    s = old + v
    vv = s - old
    err = (old - (s - vv)) + (v - vv)
    assert np.all(err[(got == 1.0) & np.isfinite(v)] == 0.0)
    assert not np.any(got[~np.isfinite(old)]) and not np.any(got[old < 0.0]) and not np.any(got[~np.isfinite(v)])
    e = lambda x: np.frexp(x)[1]
    fine = np.isfinite(old) & np.isfinite(v) & (old > 1e-300) & (v > 1e-44)
    even = (old.view(np.uint64) & np.uint64(1)) == 0
    gap = np.where(fine, e(old) - e(v), 0)
    up = fine & (gap > 0)
    assert np.array_equal(got[up] == 1.0, (gap[up] <= 28) & even[up])
    for g, last in ((0, 1), (-1, 2), (-3, 4), (-50, 51), (-51, 52), (-52, 53)):    # sh low bits of old must be 0
        at = fine & (gap == g)
        zeros = (old.view(np.uint64) & np.uint64((1 << min(last, 52)) - 1)) == 0
        assert np.array_equal(got[at] == 1.0, zeros[at] & (last <= 52)), g
    assert got[up].any() and (got[fine & (gap < -20)] == 1.0).any()


@pytest.mark.filterwarnings("ignore::RuntimeWarning")
def test_divide_by_a_known_reciprocal(host):
    a, d, got = _evaluate(host, DIVIDE, *_quotients(np.random.default_rng(2)))
    assert _same(got, a / d)


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore::RuntimeWarning")
def test_the_device_gives_the_host_s_bits(host, tmp_path):
    from mocassin_xray_gb300 import _build
    (tmp_path / "t.cu").write_text(SOURCE)
    subprocess.run([_build._nvcc(), *_build.GENCODE, "-O3", "--fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    "-I", str(CSRC), "t.cu", "-o", "t.so"], cwd=tmp_path, check=True)
    f = ctypes.CDLL(str(tmp_path / "t.so")).device
    f.restype = ctypes.c_int
    for what in range(6):
        rng = np.random.default_rng(10 + what)
        x = _sums(rng) if what == EXACT else _quotients(rng) if what == DIVIDE else _arguments(what, rng)
        assert _same(_evaluate(f, what, *x)[2], _evaluate(host, what, *x)[2]), what
