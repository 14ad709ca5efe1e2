"""The double-float functions of the generated kernels, compiled for the host
from a kernel's own source and compared with 64-bit-significand arithmetic."""
import subprocess

import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import lower_source

SHIM = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
using std::isinf;
#define __device__
#define __forceinline__ inline
#define __noinline__
#define __restrict__
struct float2 { float x, y; };
struct float4 { float x, y, z, w; };
template <class T, class S> static inline T as(S s) { T t; std::memcpy(&t, &s, sizeof t); return t; }
static inline float __int_as_float(int i) { return as<float>(i); }
static inline float __uint_as_float(unsigned i) { return as<float>(i); }
static inline unsigned __float_as_uint(float f) { return as<unsigned>(f); }
static inline int __float_as_int(float f) { return as<int>(f); }
static inline long long __double_as_longlong(double d) { return as<long long>(d); }
static inline double __longlong_as_double(long long i) { return as<double>(i); }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline float __frcp_rn(float a) { return 1.0f / a; }
static inline float __double2float_rn(double x) { return (float)x; }
static inline int __float2int_rn(float x) { return (int)lrintf(x); }
static inline float __shfl_xor_sync(unsigned, float a, int) { return a; }
// within two units in the last place, as CUDA's
static inline float rsqrtf(float x) {
  static unsigned s = 1;
  s = s * 1664525u + 1013904223u;
  return as<float>(as<unsigned>((float)(1.0 / sqrt((double)x))) + (s >> 30) % 4u - 2u);
}
"""

MAINS = {
    # relative error of sqrt over the exponents whose low word is a normal number
    "sqrt": ("""double y = exp((drand48() - 0.5) * 120); mf_dw a = mf_dw_split_rn(y), r = mf_dw_sqrt(a);
      long double t = sqrtl((long double)a.h + a.l); e = fabs((double)(((long double)r.h + r.l - t) / t));""", 2.0**-48),
    # absolute error of sin and cos over a few periods (the argument's own 2^-49 included)
    "sincos": ("""mf_dw a = mf_dw_split_rn((drand48() * 2 - 1) * 12.6), s, c; mf_dw_sincos(a, &s, &c);
      long double x = (long double)a.h + a.l;
      e = fmax(fabs((double)((long double)s.h + s.l - sinl(x))), fabs((double)((long double)c.h + c.l - cosl(x))));""",
               12.6 * 2.0**-49 + 2.0**-48),
    # a normalized pair to FP64, in units of the last place: correctly rounded; powers of two among the high words
    "to_double": ("""float h = (float)(exp((drand48() - 0.5) * 170) * (i & 1 ? -1 : 1)); if (i % 5 == 0) h = ldexpf(i & 1 ? -1 : 1, i % 250 - 125);
      float l = (float)((drand48() - 0.5) * ldexp(1.0, ilogbf(h) - 23)); if (i % 7 == 0) l = ldexpf(l, -(i % 60)); if (i % 11 == 0) l = 0;
      mf_dw p = mf_fast_two_sum(h, l); double t = (double)p.h + (double)p.l;
      e = fabs(mf_dw_to_double_bits(p) - t) / ldexp(1.0, ilogb(t) - 52); if (fabsf(h) < 1e-30f) e = 0;""", 0.0),
}


@pytest.mark.parametrize("name", sorted(MAINS))
def test_double_float_function(name, tmp_path):
    src = lower_source("k", L.MF_KERNEL_STORE, L.MF_F64, ["x"], [], ["sqrt(x)"])
    pre = src[src.index("#define MF_LN2_HI"):src.index('extern "C" __global__')]
    body, tol = MAINS[name]
    (tmp_path / "t.cpp").write_text(SHIM + pre + f"""
int main() {{
  double worst = 0;
  for (int i = 0; i < 400000; i++) {{ double e = 0; {body} worst = fmax(worst, e); }}
  const float inf = __int_as_float(0x7f800000);
  printf("%.17g %d\\n", worst, isinf(mf_dw_to_double_bits(mf_dw_make(-inf, 0))) && mf_dw_to_double_bits(mf_dw_make(-inf, 0)) < 0
         && std::isnan(mf_dw_to_double_bits(mf_dw_make(NAN, 0))) && mf_dw_to_double_bits(mf_dw_make(0, 0)) == 0.0
         && mf_dw_to_double_bits(mf_dw_make(1e-40f, 0)) == 0.0 && mf_dw_sqrt(mf_dw_make(0, 0)).h == 0.0f
         && std::isnan(mf_dw_sqrt(mf_dw_make(-1, 0)).h) && mf_dw_sqrt(mf_dw_make(inf, 0)).h == inf);
}}
""")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")],
                   check=True)
    worst, special = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    assert special == "1"
    assert float(worst) <= tol
