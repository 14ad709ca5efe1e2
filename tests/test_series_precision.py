"""The double-float sine and cosine, run on the host from a kernel's source:
no further from 64-bit-significand arithmetic than the same series with every
product and sum normalized."""
import subprocess

from morefit_gb300 import _lib as L
from morefit_gb300.backend import lower_source
from test_doublefloat import SHIM


def test_sine_and_cosine_are_as_accurate_as_normalized_steps(tmp_path):
    src = lower_source("k", L.MF_KERNEL_STORE, L.MF_F64, ["x"], [], ["sin(x)"])
    pre = src[src.index("#define MF_LN2_HI"):src.index('extern "C" __global__')]
    series = pre[pre.index("__device__ __forceinline__ void mf_dw_sincos"):]
    series = series[:series.index("\n}\n") + 3].replace("mf_dw_sincos", "normalized")
    series = series.replace("mf_dw_horner_last(", "step(").replace("mf_dw_horner(", "step(")
    assert series.count("step(") == 11
    (tmp_path / "t.cpp").write_text(SHIM + pre + f"""
static mf_dw step(mf_dw c, mf_dw x, mf_dw q) {{ return mf_dw_add(c, mf_dw_mul(x, q)); }}
{series}
int main() {{
  double s[4] = {{0}}, m[4] = {{0}};
  const int n = 2000000;
  for (int i = 0; i < n; i++) {{
    const mf_dw a = mf_dw_split_rn((drand48() * 2 - 1) * 0.785);
    mf_dw r[4];
    mf_dw_sincos(a, r, r + 1);
    normalized(a, r + 2, r + 3);
    const long double x = (long double)a.h + a.l, t[2] = {{sinl(x), cosl(x)}};
    for (int q = 0; q < 4; q++) {{
      const double e = (double)(((long double)r[q].h + r[q].l - t[q % 2]) / t[q % 2]);
      s[q] += e * e;
      m[q] = fmax(m[q], fabs(e));
    }}
  }}
  for (int q = 0; q < 4; q++) printf("%.17g %.17g\\n", sqrt(s[q] / n), m[q]);
}}
""")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")],
                   check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    (sr, sm, cr, cm), (nsr, nsm, ncr, ncm) = [[float(v) for v in out[4 * i:4 * i + 4]] for i in range(2)]
    # the rms of two million errors is known to 0.1%
    assert sr <= 1.001 * nsr and cr <= 1.001 * ncr, out
    assert sm <= 1.001 * nsm and cm <= 1.001 * ncm, out
