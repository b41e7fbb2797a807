"""scale_narrow's claim (its float is narrow(x * r) wherever it says so) holds whichever products and sums the compiler
contracts: its source, built for the host on a float type whose every product stays open to contraction into the sums
that read it, against the two exact roundings."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from pycompute_gb300 import build

SHIM = r"""
#include <cmath>
#include <cstdint>
#include <cstring>
#define PCGB_HD static inline
template <class T, class F> static inline T as(F f) { T t; std::memcpy(&t, &f, sizeof(t)); return t; }
// A float that remembers the product it came from; a sum fuses one of its operands' products.
struct contracted {
  float v = 0, a = 0, b = 0;
  bool product = false;
  contracted() = default;
  contracted(float x) : v(x) {}
};
static contracted operator-(contracted x) { x.v = -x.v; x.a = -x.a; return x; }
static contracted operator*(contracted x, contracted y) {
  contracted r(x.v * y.v);
  r.a = x.v;
  r.b = y.v;
  r.product = true;
  return r;
}
static contracted operator+(contracted x, contracted y) {
  if (RIGHT ? y.product : !x.product && y.product) return std::fmaf(y.a, y.b, x.v);
  if (x.product) return std::fmaf(x.a, x.b, y.v);
  return x.v + y.v;
}
static contracted operator-(contracted x, contracted y) { return x + -y; }
static bool operator==(contracted x, contracted y) { return x.v == y.v; }
static bool operator<(contracted x, contracted y) { return x.v < y.v; }
static bool operator>(contracted x, contracted y) { return x.v > y.v; }
static contracted fabsf(contracted x) { return std::fabs(x.v); }
static contracted fmaf(contracted x, contracted y, contracted z) { return std::fmaf(x.v, y.v, z.v); }
// the device's operations that are never contracted
static contracted __fmul_rn(contracted x, contracted y) { return x.v * y.v; }
static contracted __fadd_rn(contracted x, contracted y) { return x.v + y.v; }
static void words(double x, unsigned& lo, unsigned& hi) {
  const uint64_t b = as<uint64_t>(x);
  lo = unsigned(b);
  hi = unsigned(b >> 32);
}
static unsigned __funnelshift_l(unsigned lo, unsigned hi, unsigned s) {
  return unsigned(((uint64_t(hi) << 32 | lo) << s) >> 32);
}
static contracted __uint_as_float(unsigned u) { return as<float>(u); }
"""


@pytest.mark.parametrize("right", [0, 1])
def test_scale_narrow_is_exact_under_any_contraction(tmp_path, right):
    src = open(os.path.join(build.CSRC, "lm_kernel.cuh")).read()
    body = re.search(r"^PCGB_HD bool scale_narrow\(.*?^}\n", src, re.S | re.M).group(0)
    (tmp_path / "t.cpp").write_text(f"#define RIGHT {right}\n{SHIM}#define float contracted\n{body}#undef float\n" + r"""
extern "C" void run(const double* x, const float* r, float* out, int* ok, long n) {
  for (long i = 0; i < n; ++i) {
    contracted o;
    ok[i] = scale_narrow(x[i], r[i], o);
    out[i] = o.v;
  }
}
""")
    lib = str(tmp_path / "t.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", str(tmp_path / "t.cpp"), "-o",
                    lib], check=True)
    rng = np.random.default_rng(11)
    n = 1 << 20
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-25, 25, n)) * rng.choice([-1.0, 1.0], n)
    r = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-30, 30, n)).astype(np.float32)
    out, ok = np.empty(n, np.float32), np.empty(n, np.int32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    ctypes.CDLL(lib).run(p(x), p(r), p(out), p(ok), ctypes.c_long(n))
    told = ok != 0
    assert told.mean() > 0.99
    want = (x * r.astype(np.float64)).astype(np.float32)
    np.testing.assert_array_equal(out.view(np.int32)[told], want.view(np.int32)[told])
