"""Sums of products in the double-float event loop, taken from the generated
source and run on the host: their error against 64-bit-significand arithmetic
is no larger than that of normalized products and normalized additions."""
import re
import subprocess

import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import lower_source
from test_doublefloat import SHIM

N = "mf_dw_neg"
# text, the same by normalized operations, the value in long double, its terms' magnitudes
SUMS = {
    "two products and a value": ("((x*y)+(z*x)+v)", "A(A(M(x,y),M(z,x)),v)", "x*y+z*x+v", "x*y+z*x+v"),
    "two products": ("((x*y)+(z*v))", "A(M(x,y),M(z,v))", "x*y+z*v", "x*y+z*v"),
    "a difference of products": ("((x*y)+-((z*v)))", f"A(M(x,y),{N}(M(z,v)))", "x*y-z*v", "x*y+z*v"),
    "a product and two values": ("((x*y)+z+v)", "A(A(M(x,y),z),v)", "x*y+z+v", "x*y+z+v"),
    "three products": ("((x*y)+(z*v)+(x*v))", "A(A(M(x,y),M(z,v)),M(x,v))", "x*y+z*v+x*v", "x*y+z*v+x*v"),
}


@pytest.mark.parametrize("name", sorted(SUMS))
@pytest.mark.parametrize("output", [False, True], ids=["statement", "output"])
def test_sum_is_as_accurate_as_normalized_operations(name, output, tmp_path):
    text, normal, value, magnitude = SUMS[name]
    src = lower_source("k", L.MF_KERNEL_REDUCE, L.MF_F64, ["x", "y", "z", "v"], [],
                       [text if output else f"sqrt({text})"], vec=1)
    store = lower_source("k", L.MF_KERNEL_STORE, L.MF_F64, ["x"], [], ["sqrt(x)"])
    pre = store[store.index("#define MF_LN2_HI"):store.index('extern "C" __global__')]
    part = src[src.index("mf_reduce_part("):]
    cols = [re.search(rf"//   y(\d+) = \+ 1\*{c}\n", src).group(1) for c in "xyzv"]
    body = re.search(r"(?:const mf_dw x\d+ = .*\n\s*)+((?:.*\n)*?)\s*\}\n  \}\n", part).group(1)
    body = body.replace("if (base + 0 < n)", "")
    if not output:  # up to the square root: its operand
        at, operand = body.index("= mf_dw_sqrt("), re.search(r"mf_dw_sqrt\((\w+)\)", body).group(1)
        body = body[:body.rindex("\n", 0, at) if "\n" in body[:at] else 0] + f"\nacc[0] = {operand};"
    (tmp_path / "t.cpp").write_text(SHIM + pre + f"""
static mf_dw A(mf_dw a, mf_dw b) {{ return mf_dw_add(a, b); }}
static mf_dw M(mf_dw a, mf_dw b) {{ return mf_dw_mul(a, b); }}
static mf_dw draw() {{ return mf_dw_split_rn(0.5 + 1.5 * drand48()); }}
typedef long double ld;
static ld V(mf_dw a) {{ return (ld)a.h + a.l; }}
static mf_dw kernel(mf_dw x{cols[0]}, mf_dw x{cols[1]}, mf_dw x{cols[2]}, mf_dw x{cols[3]}) {{
  mf_dw acc[1] = {{mf_dw_make(0.0f, 0.0f)}};
  {body}
  return mf_dw_renorm(acc[0]);
}}
int main() {{
  double s[2] = {{0, 0}};
  for (int i = 0; i < 400000; i++) {{
    const mf_dw a = draw(), b = draw(), c = draw(), d = draw();
    const mf_dw r[2] = {{kernel(a, b, c, d), [](mf_dw x, mf_dw y, mf_dw z, mf_dw v) {{ return {normal}; }}(a, b, c, d)}};
    const ld x = V(a), y = V(b), z = V(c), v = V(d), t = {value}, m = {magnitude};
    for (int q = 0; q < 2; q++) {{ const double e = (double)((V(r[q]) - t) / m); s[q] += e * e; }}
  }}
  printf("%.17g %.17g\\n", sqrt(s[0] / 400000), sqrt(s[1] / 400000));
}}
""")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")],
                   check=True)
    got, ref = map(float, subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split())
    # the rms of 400000 errors is known to about 0.2%
    assert got <= 1.01 * ref, (got, ref)
