"""The stage kernels' own quotients (csrc/quotient.cuh) against plain division, bit for bit,
over the operands where they could go wrong: quotients within a hair of a rounding tie, both
ends of the range of exponents, significands of all ones, zeros, infinities and NaN.  What
they cannot answer they must say (`bad`), and nothing else."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from storm_b200 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include "quotient.cuh"
using namespace storm;
__global__ void k_quot(const double* a, const double* b, int n, double* q, double* e, unsigned char* bad) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool x = false;
  q[i] = Den<double>(b[i], &x).quot(a[i], &x);
  e[i] = fabs(__fma_rn(-b[i], Den<double>::seed(b[i]), 1.0));
  bad[i] = x;
}
__global__ void k_lim(const double* f, int n, double* r, unsigned char* bad) {  // f: q0, then per face qn, gx, gy, rx, ry
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool x = false;
  Limit3<double> l;
  for (int k = 0; k < 3; k++) {
    const double* p = f + (size_t)(1 + 5 * k) * n + i;
    l.face(f[i], p[0], p[n], p[2 * (size_t)n], p[3 * (size_t)n], p[4 * (size_t)n], &x);
  }
  r[i] = l.value(&x);
  bad[i] = x;
}
template <class F>
static int with_device(const void* const* in, const size_t* nin, int kin, void* const* out, const size_t* nout, int kout, F run) {
  void* p[8] = {};
  int rc = 0;
  for (int i = 0; i < kin + kout; i++) rc |= cudaMalloc(&p[i], i < kin ? nin[i] : nout[i - kin]);
  for (int i = 0; i < kin && !rc; i++) rc |= cudaMemcpy(p[i], in[i], nin[i], cudaMemcpyHostToDevice);
  if (!rc) run(p);
  if (!rc) rc = cudaDeviceSynchronize();
  for (int i = 0; i < kout && !rc; i++) rc |= cudaMemcpy(out[i], p[kin + i], nout[i], cudaMemcpyDeviceToHost);
  for (int i = 0; i < kin + kout; i++) cudaFree(p[i]);
  return rc;
}
extern "C" __attribute__((visibility("default"))) int quot(const double* a, const double* b, int n, double* q, double* e, unsigned char* bad) {
  const void* in[] = {a, b};
  const size_t w = 8 * (size_t)n, nin[] = {w, w}, nout[] = {w, w, (size_t)n};
  void* out[] = {q, e, bad};
  return with_device(in, nin, 2, out, nout, 3, [&](void** p) {
    k_quot<<<(n + 255) / 256, 256>>>((double*)p[0], (double*)p[1], n, (double*)p[2], (double*)p[3], (unsigned char*)p[4]);
  });
}
extern "C" __attribute__((visibility("default"))) int lim(const double* f, int n, double* r, unsigned char* bad) {
  const void* in[] = {f};
  const size_t w = 8 * (size_t)n, nin[] = {16 * w}, nout[] = {w, (size_t)n};
  void* out[] = {r, bad};
  return with_device(in, nin, 1, out, nout, 2, [&](void** p) {
    k_lim<<<(n + 255) / 256, 256>>>((double*)p[0], n, (double*)p[1], (unsigned char*)p[2]);
  });
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    if not shutil.which(build.nvcc()):
        pytest.skip("compiles its probe: needs nvcc")
    d = tmp_path_factory.mktemp("quotient")
    (d / "probe.cu").write_text(SRC)
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", build.CSRC, "-shared", "-o", str(d / "probe.so"),
                    str(d / "probe.cu")], check=True, cwd=d, capture_output=True)
    return ctypes.CDLL(os.path.join(d, "probe.so"))


def _vp(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _quot(probe, a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    q, e, bad = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.uint8)
    assert probe.quot(_vp(a), _vp(b), a.size, _vp(q), _vp(e), _vp(bad)) == 0
    with np.errstate(all="ignore"):
        r = a / b
    good = bad == 0
    assert np.array_equal(q[good].view(np.uint64), r[good].view(np.uint64))
    return good, e


def _random(rng, n, lo, hi):
    m = rng.integers(1 << 52, 1 << 53, size=n).astype(np.float64)
    return np.ldexp(m * rng.choice([-1.0, 1.0], size=n), rng.integers(lo, hi, size=n) - 52)


def _ones(x):
    return (x.view(np.uint64) & np.uint64((1 << 52) - 1)) == np.uint64((1 << 52) - 1)


@pytest.mark.parametrize("lo,hi", [(-450, 451), (-3, 4)])
def test_random_quotients(lo, hi, probe):
    rng = np.random.default_rng(5)
    a, b = _random(rng, 4_000_000, lo, hi), _random(rng, 4_000_000, lo, hi)
    good, e = _quot(probe, a, b)
    assert (good | _ones(b)).all()  # every ordinary pair is answered
    assert e.max() < 2.0 ** -17  # the seed, as the derivation takes it


def test_near_ties(probe):
    """2^54 a = r + m b with an odd m and a small r: a / b lies r / (2^54 b) beside the middle
    of two neighbouring numbers."""
    rng = np.random.default_rng(6)
    a, b = [], []
    while len(a) < 20000:
        y = int(rng.integers(1 << 52, 1 << 53)) | 1
        inv = pow(1 << 54, -1, y)
        for r in (-3, -2, -1, 1, 2, 3):
            x = r * inv % y
            if 2 * x >= y and ((x << 54) - r) // y % 2 == 1:
                a.append(float(x))
                b.append(float(y))
    good, _ = _quot(probe, a, b)
    assert (good | _ones(np.array(b))).all()


def test_quotients_left_to_the_division(probe):
    ones = np.ldexp(2.0 - 2.0 ** -52, [-450, -1, 0, 1, 450])
    for b in ones:  # all ones: whatever the numerator
        assert not _quot(probe, [1.0, -3.0, 0.0, b], [b] * 4)[0].any()
    edge = [2.0 ** -450, -(2.0 ** -450), np.nextafter(2.0 ** 451, 0.0) - 2.0 ** 399, 2.0 ** 450]
    out = [np.nextafter(2.0 ** -450, 0.0), 2.0 ** 451, -(2.0 ** 500), 1e-320, np.inf, -np.inf, np.nan]
    for x in edge:
        for y in edge:
            assert _quot(probe, [x, 0.0, -0.0], [y] * 3)[0].all()
    for x in out + [0.0, -0.0]:
        assert not _quot(probe, [1.0, 0.0, x], [x] * 3)[0].any()
    for x in out:
        assert not _quot(probe, [x, x], [3.0, -0.7])[0].any()


def _ratios(f):
    """The least of the three ratios as the expressions say it (limiterBJ.f90:42-81)."""
    q0, least = f[0], None
    with np.errstate(all="ignore"):
        for k in range(3):
            qn, gx, gy, rx, ry = f[1 + 5 * k:6 + 5 * k]
            qmin, qmax = np.where(qn < q0, qn, q0), np.where(qn > q0, qn, q0)
            delq = (q0 + gx * rx + gy * ry) - q0
            eps = np.abs(delq) * 2.0 ** -52
            eps = np.where(eps == 0, 2.0 ** -1022, eps)
            num = np.where(delq < 0, qmin - q0, qmax - q0)
            r = np.where(~(np.abs(delq) > eps) | (np.abs(num) > np.abs(delq)), 1.0, num / delq)
            r = np.where(1.0 < r, 1.0, r)
            least = r if least is None else np.where(r < least, r, least)
    return least


def _limit(probe, f):
    f = np.ascontiguousarray(f, np.float64)
    r, bad = np.empty(f.shape[1]), np.empty(f.shape[1], np.uint8)
    assert probe.lim(_vp(f), f.shape[1], _vp(r), _vp(bad)) == 0
    good = bad == 0
    assert np.array_equal(r[good].view(np.uint64), _ratios(f)[good].view(np.uint64))
    return good


def _faces(rng, n, q0, step):
    f = np.empty((16, n))
    f[0] = q0
    for k in range(3):
        f[1 + 5 * k] = q0 + step * rng.normal(size=n)
        f[2 + 5 * k:4 + 5 * k] = step * rng.normal(size=(2, n))
        f[4 + 5 * k:6 + 5 * k] = rng.uniform(-1.0, 1.0, size=(2, n))
    return f


@pytest.mark.parametrize("q0,step", [(1.0, 1e-2), (1.0, 1e-14), (0.0, 1.0), (0.0, 1e-100), (-300.0, 5.0)])
def test_limiter(q0, step, probe):
    good = _limit(probe, _faces(np.random.default_rng(7), 1_000_000, q0, step))
    assert good.mean() > (0.999 if step > 1e-10 or q0 == 0.0 else 0.0)


@pytest.mark.parametrize("step", [1e-138, 1e-144, 1e-145, 1e-146, 1e-150, 1e-160, 1e-300, 1e-308, 1e-320, 1e150, 1e160, 1e300])
def test_limiter_out_of_range(step, probe):
    """Cross products around 1e-290, subnormal and infinite."""
    _limit(probe, _faces(np.random.default_rng(8), 300_000, 0.0, step))


def test_limiter_ties(probe):
    """Two faces with one ratio, or ratios some units in the last place apart; still water;
    infinities and NaN in any place."""
    rng = np.random.default_rng(9)
    n = 500_000
    f = _faces(rng, n, 0.0, 1.0)
    near = f.copy()
    s = np.ldexp(rng.choice([-1.0, 1.0], size=n), rng.integers(-3, 4, size=n))
    near[6:9] = f[1:4] * s  # face 1: face 0's values times a power of two
    near[9:11] = f[4:6]
    _limit(probe, near)
    near[6] *= 1.0 + rng.integers(-20, 21, size=n) * 2.0 ** -52
    _limit(probe, near)
    still = f * rng.integers(0, 2, size=f.shape)
    _limit(probe, still)
    wild = f.copy()
    hit = rng.random(f.shape) < 0.05
    wild[hit] = rng.choice([np.inf, -np.inf, np.nan, 1e308, 5e-324, -0.0], size=int(hit.sum()))
    _limit(probe, wild)
