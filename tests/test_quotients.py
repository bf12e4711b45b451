"""quotients() of csrc/quotients.cuh (several FP64 quotients by one reciprocal) against the division, compiled
for the CPU: its operations are IEEE ones, so the CPU's fma and division give what the device gives.  Every
quotient has to be the division's, down to the sign of a zero: a vertical Courant number is formed this
way, and the limiter reads its inflow side from the sign."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "icoatmosbenchmark_v1_b200" / "csrc"

SHIM = r"""
#include <cmath>
#include <cstring>
#define __device__
#define __forceinline__ inline
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline int __double2hiint(double x) {
  unsigned long long u;
  std::memcpy(&u, &x, 8);
  return (int)(u >> 32);
}
#include "quotients.cuh"
extern "C" void shared(long n, const double *a, const double *b, double *q) {
  for (long i = 0; i < n; ++i) {
    double x[2] = {a[2 * i], a[2 * i + 1]};
    icoadv::quotients(x, icoadv::recip(b[i]));
    q[2 * i] = x[0], q[2 * i + 1] = x[1];
  }
}
"""


@pytest.fixture(scope="module")
def shared(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("quotients")
    (d / "q.cpp").write_text(SHIM)
    subprocess.run([cxx, "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-Wno-unknown-pragmas", f"-I{CSRC}",
                    str(d / "q.cpp"), "-o", str(d / "q.so")], check=True)
    fn = C.CDLL(str(d / "q.so")).shared

    def run(a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        q = np.empty_like(a)
        p = lambda x: x.ctypes.data_as(C.c_void_p)  # noqa: E731
        fn(C.c_long(b.size), p(a), p(b), p(q))
        return q

    return run


def _same(q, a, b):
    with np.errstate(all="ignore"):
        want = a / b[:, None]
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(q), nan)
    bad = (q.view(np.int64) != want.view(np.int64)) & ~nan
    assert not bad.any(), (a[bad][:4], np.broadcast_to(b[:, None], a.shape)[bad][:4], q[bad][:4], want[bad][:4])


EDGES = [0.0, 5e-324, 2.0**-1022, 2.0**-900, 2.0**-801, 2.0**-800, 2.0**-101, 2.0**-100, 1.0 / 3.0, 1.0, 1.0 + 2.0**-52,
         2.0 - 2.0**-52, 2.0**100, 2.0**101, 2.0**999, 2.0**1000, np.finfo(np.float64).max, np.inf, np.nan]


def test_every_pair_of_edges_and_signs(shared):
    e = np.array(EDGES + [-x for x in EDGES])
    a0, a1, b = (x.ravel() for x in np.meshgrid(e, e, e, indexing="ij"))
    a = np.stack([a0, a1], axis=1)
    _same(shared(a, b), a, b)


def test_signed_zero_beside_ordinary_dividends(shared):
    rng = np.random.default_rng(1)
    b = rng.uniform(0.1, 2.0, 2000) * rng.choice([-1.0, 1.0], 2000)
    a = np.stack([rng.standard_normal(2000), rng.choice([-0.0, 0.0], 2000)], axis=1)
    _same(shared(a, b), a, b)


def test_random_magnitudes(shared):
    rng = np.random.default_rng(2)
    n = 200000
    b = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-110, 110, n)) * rng.choice([-1.0, 1.0], n)
    a = np.ldexp(rng.uniform(1.0, 2.0, (n, 2)), rng.integers(-950, 1000, (n, 2))) * rng.choice([-1.0, 1.0], (n, 2))
    _same(shared(a, b), a, b)
