"""The event loop of the ragged-segment entries, taken from the generated
source and run on the host: every event once, nothing read outside the segment,
and an end, for segments of every size that a 32-bit count holds."""
import re
import subprocess

import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import lower_source


def _loop(src, entry):
    """(loop header, declarations in the loop, [(condition, event) of each load ahead])."""
    t = src[src.index(f"mf_reduce{entry}("):]
    t = t[:t.index("__shared__ float2 mf_part")]
    m = re.search(r"\n  for \((\w+ i = threadIdx\.x; .*?)\) \{\n(.*)\n  \}\n", t, re.S)
    decls = re.findall(r"^    const (?:unsigned|mf_u64|bool) \w+ = .*;$", m.group(2), re.M)
    ahead = re.findall(r"^    c\d+ = (.*) \? __ldg\(data \+ \(mf_u64\)\d+ \* stride \+ first \+ (.*)\) :", m.group(2), re.M)
    return m.group(1), decls, ahead


@pytest.mark.parametrize("elem", [L.MF_F64, L.MF_F32])
@pytest.mark.parametrize("entry", ["_segments", "_multi"])
def test_segment_loop_ends(elem, entry, tmp_path):
    header, decls, ahead = _loop(lower_source("k", L.MF_KERNEL_REDUCE, elem, ["x"], ["a"], ["log((a*x))"]), entry)
    assert bool(ahead) == (elem == L.MF_F64)
    loads = "".join(f"if ({c}) {{ bad |= (mf_u64)({e}) >= cnt || (mf_u64)({e}) != i + MF_BLOCK; }}" for c, e in ahead)
    (tmp_path / "t.cpp").write_text(f"""#include <cstdio>
#include <initializer_list>
typedef unsigned long long mf_u64;
constexpr unsigned MF_BLOCK = 256;
struct {{ unsigned x; }} threadIdx;
int main() {{
  const unsigned counts[] = {{0u, 1u, 255u, 256u, 257u, 513u, 0xfffffeffu, 0xffffff00u, 0xffffff01u, 0xffffffffu}};
  for (unsigned cnt : counts)
    for (unsigned t : {{0u, 1u, 254u, 255u}}) {{
      threadIdx.x = t;
      const mf_u64 want = cnt > t ? (cnt - t + (mf_u64)MF_BLOCK - 1) / MF_BLOCK : 0;
      mf_u64 turns = 0;
      bool bad = false;
      for ({header}) {{
        bad |= i != t + turns * MF_BLOCK;
        {" ".join(decls)} {loads}
        if (++turns > want) break;
      }}
      if (bad || turns != want) {{ printf("count %u thread %u: %llu turns for %llu\\n", cnt, t, turns, want); return 1; }}
    }}
  return 0;
}}
""")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
