"""Accept-reject generation: the FP32 accept test's error bound (CPU) and the
events of the cooperative generator at the edges of its launch rule (GPU)."""
import ctypes as C
import re
import subprocess

import numpy as np
import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import lower_source
from morefit_gb300.workloads import load_spec

SHIM = """
#include <cmath>
#include <cstring>
#define __device__
#define __forceinline__ inline
static inline float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
static inline float __frcp_rn(float x) { return 1.0f / x; }
static inline float rsqrtf(float x) { return 1.0f / sqrtf(x); }
"""

# every operation of the kernel language, with its poles and branches in range
ALL_OPS = ("(2.0+sin((3.0*x))*cos(y)+sin(y)+tan((0.7*x))*0.1+asin((0.9*x))+acos((y*0.9))+atan((x*y))+erf((x-y))"
           "+exp((x*y))+0.01*log((1.5+x*y))+sqrt((1.0-(x*x)))+pow((1.2+y),2.5)+pow((1.5+x),(y+3.0))"
           "+1.0/((2.5+x))+(((x+0.25)>0.0) ? (x*y) : ((y==0.0) ? 1.0 : (-(y)*a))))/25.0")


def _numpy(text, values):
    """The expression in 64 bits: C conditionals as nested np.where calls."""
    def conv(t):
        stack, out = [], ""
        for ch in t:
            if ch == "(":
                stack.append((out, []))
                out = ""
            elif ch in "?:":
                stack[-1][1].append(out)
                out = ""
            elif ch == ")":
                before, parts = stack.pop()
                out = before + ("np.where(%s,%s,%s)" % (*parts, out) if parts else "(" + out + ")")
            else:
                out += ch
        return out
    from math import erf
    names = {"np": np, "pow": np.power, "asin": np.arcsin, "acos": np.arccos, "atan": np.arctan,
             "erf": np.vectorize(erf), **{f: getattr(np, f) for f in ("sin", "cos", "tan", "exp", "log", "sqrt")}}
    return eval(conv(text), {**names, **values})


def _cases():
    for m in ("mass", "pwave", "cbpoly", "spwave"):
        g = next(k for k in load_spec(m)["kernels"] if k.get("generate"))
        yield m, g["exprs"][0], g["outputs"], g["lo"], g["hi"], g["maxprob"], {}
    yield "all operations", ALL_OPS, ["x", "y"], [-1.0, -1.0], [1.0, 1.0], 1.0, {"a": 0.7}


@pytest.mark.parametrize("case", list(_cases()), ids=lambda c: c[0])
def test_fp32_density_bound_holds(case, tmp_path):
    """The generator decides in FP32 where |maxprob u - p| exceeds the bound:
    the bound holds at every sampled point, and is tight enough that almost
    every decision is made in FP32."""
    name, expr, dims, lo, hi, maxprob, par = case
    src = lower_source("g", L.MF_KERNEL_GENERATE, L.MF_F64, [], list(par), [expr], gen=(dims, lo, hi, maxprob))
    code = src[src.index("struct mf_ef "):src.index("extern \"C\" __global__")]
    sig = re.search(r"mf_filter\((.*)bool& amb\)", code).group(1)
    uni = re.findall(r"mf_ef uf(\d+)", sig)
    assert len(uni) == len(par)
    args = ", ".join(f"mf_ef_make(v[{d}], e[{d}])" for d in range(len(dims)))
    args += "".join(f", mf_ef_from(u[{i}])" for i in range(len(uni)))
    (tmp_path / "f.cpp").write_text(SHIM + code + f"""
extern "C" void run(int n, const float* xs, const float* e, const double* u, float* p, float* q, unsigned char* amb) {{
  for (int i = 0; i < n; i++) {{
    const float* v = xs + i * {len(dims)};
    bool a = false;
    const mf_ef r = mf_filter({args}, a);
    p[i] = r.v; q[i] = r.e; amb[i] = a;
  }}
}}
""")
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-o", str(tmp_path / "f.so"), str(tmp_path / "f.cpp")], check=True)
    lib = C.CDLL(str(tmp_path / "f.so"))
    n = 200000
    rng = np.random.default_rng(3)
    lo, hi = np.array(lo, float), np.array(hi, float)
    draws = rng.integers(0, 2**32, (n, len(dims)), dtype=np.uint64).astype(np.float64)
    draws[:64] = rng.choice([0.0, 1.0, 2.0**32 - 1, 2.0**31, 2.0**31 - 1], (64, len(dims)))
    x = lo + (hi - lo) * (draws * 2.0**-32)
    # as the kernel forms them: one fused multiply-add of FP32 constants
    u32 = draws.astype(np.float32).astype(np.float64) * 2.0**-32
    xs = np.ascontiguousarray((u32 * np.float64(np.float32(hi - lo)) + np.float64(np.float32(lo))).astype(np.float32))
    e = ((np.abs(lo) + np.abs(hi - lo)) * 2.0**-22).astype(np.float32)
    u = np.array([par[k] for k in par] or [0.0])
    p, q, amb = np.zeros(n, np.float32), np.zeros(n, np.float32), np.zeros(n, np.uint8)
    lib.run(n, xs.ctypes.data_as(C.c_void_p), e.ctypes.data_as(C.c_void_p), u.ctypes.data_as(C.c_void_p),
            p.ctypes.data_as(C.c_void_p), q.ctypes.data_as(C.c_void_p), amb.ctypes.data_as(C.c_void_p))
    with np.errstate(all="ignore"):
        ref = _numpy(expr, {**{d: x[:, i] for i, d in enumerate(dims)}, **par})
    sure = (amb == 0) & np.isfinite(q) & np.isfinite(p)
    assert np.isfinite(ref[sure]).all()
    assert (np.abs(p[sure].astype(np.float64) - ref[sure]) <= 1.01 * q[sure].astype(np.float64)).all()
    assert sure.mean() > 0.99 and np.median(q[sure]) < 1e-4 * maxprob


@pytest.mark.parametrize("nrows,seed", [(1, 0), (2, 2**64 - 1), (257, 229387429), (8192, 12345)])
def test_seed_rows_equal_the_stepped_jumps(nrows, seed):
    """The table-driven jump gives the rows that stepping through the jump
    polynomial gives (the C restatement)."""
    from morefit_gb300.workloads import seed_rows
    from oracle import mforacle
    assert np.array_equal(seed_rows(nrows, seed), mforacle.seed_rows(nrows, seed))


@pytest.mark.gpu
@pytest.mark.parametrize("workload", ["mass", "pwave"])
@pytest.mark.parametrize("n", [1, 31, 1671, 1673, 6689, 8192, 8193, 100003])
def test_events_equal_the_streams(workload, n):
    """32, 16, 8 lanes a stream, ragged last warps and streams: bit for bit
    the events of one thread walking each stream (the C restatement)."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import generate_events, generate_partition
    from oracle import mforacle
    b = CUDABackend(0)
    cols = generate_events(b, load_spec(workload), n, seed=mforacle.SEED)
    nper, nseeds = generate_partition(n)
    assert np.array_equal(cols.download(), mforacle.generate_partitioned(workload, n, nper, nseeds))
    b.close()


@pytest.mark.gpu
def test_max_tries_counts_proposals():
    """A stream gives up after exactly max_tries proposals, whatever its lanes:
    the smallest limit that succeeds is the number of proposals the slowest
    stream needs."""
    from morefit_gb300._lib import MFError
    from morefit_gb300.backend import CUDABackend, CUDABlock
    from morefit_gb300.workloads import seed_rows
    from oracle import mforacle
    b = CUDABackend(0)
    gk = next(k for k in load_spec("mass")["kernels"] if k.get("generate"))
    blk = CUDABlock(b, np.float64)
    blk.MakeGenerateKernel(gk["name"], 40, [], gk["outputs"], gk["params"], gk["exprs"], gk["maxprob"],
                           ranges=list(zip(gk["lo"], gk["hi"])))
    blk.CopyToSeedBuffer(seed_rows(2, mforacle.SEED))
    blk.SetNevents(40)
    fails = []
    for limit in range(20, 4000):
        try:
            blk.SubmitKernel(nper=20, max_tries=limit)
        except MFError:
            fails.append(limit)
            continue
        break
    # proposals of each stream by the oracle's own walk of the same streams
    need = 0
    for t in range(2):
        s = [int(v) for v in seed_rows(2, mforacle.SEED)[:, t]]
        got = tries = 0
        events = mforacle.generate_partitioned("mass", 40, 20, 2)[0, 20 * t:20 * t + 20]
        rotl = lambda x, k: ((x << k) | (x >> (32 - k))) & 0xFFFFFFFF  # noqa: E731

        def draw():
            r = (rotl((s[0] + s[3]) & 0xFFFFFFFF, 7) + s[0]) & 0xFFFFFFFF
            w = (s[1] << 9) & 0xFFFFFFFF
            s[2] ^= s[0]
            s[3] ^= s[1]
            s[1] ^= s[2]
            s[0] ^= s[3]
            s[2] ^= w
            s[3] = rotl(s[3], 11)
            return r
        while got < 20:
            x = 5000.0 + 600.0 * (draw() * 2.3283064365386963e-10)
            draw()
            tries += 1
            got += x == events[got]
        need = max(need, tries)
    assert limit == need and len(fails) == need - 20
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("elem", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("dims,nper,streams", [(1, 23, 3), (1, 24, 3), (2, 47, 5), (7, 48, 3), (24, 30, 2), (25, 30, 2),
                                               (2, 24, 3400), (1, 48, 1700)])
def test_runs_of_proposals_equal_the_streams(dims, nper, streams, elem):
    """Several proposals a thread and turn (8, 6 and 2 of them, in 8, 16 and 32
    lanes) and the lengths around the rule: the events of one thread walking
    each stream, here in Python, and the smallest proposal limit that succeeds
    is the longest walk."""
    from morefit_gb300._lib import MFError
    from morefit_gb300.backend import CUDABackend, CUDABlock
    from morefit_gb300.workloads import seed_rows
    n = streams * nper - 1
    seeds = seed_rows(streams, 77)
    s = [seeds[k].astype(np.uint64) for k in range(4)]
    m32 = np.uint64(0xFFFFFFFF)
    rotl = lambda x, k: ((x << np.uint64(k)) | (x >> np.uint64(32 - k))) & m32  # noqa: E731

    def draw():
        r = (rotl((s[0] + s[3]) & m32, 7) + s[0]) & m32
        w = (s[1] << np.uint64(9)) & m32
        s[2] ^= s[0]
        s[3] ^= s[1]
        s[1] ^= s[2]
        s[0] ^= s[3]
        s[2] ^= w
        s[3] = rotl(s[3], 11)
        return r.astype(elem) * elem(2.0**-32)
    want = np.zeros((dims, n), elem)
    got = np.zeros(streams, np.int64)
    quota = np.minimum(nper, n - nper * np.arange(streams))
    tries = 0
    while (got < quota).any():
        x = np.array([draw() for _ in range(dims)])
        # the density x0 * x_last is exact enough in either type that no
        # decision of these streams is a tie
        take = (draw() < x[0] * x[-1]) & (got < quota)
        at = nper * np.arange(streams) + got
        want[:, at[take]] = x[:, take]
        got += take
        tries += 1
    names = [f"x{d}" for d in range(dims)]
    b = CUDABackend(0)
    blk = CUDABlock(b, elem)
    blk.MakeGenerateKernel("g", n, [], names, [], [f"(x0*{names[-1]})"], 1.0, ranges=[(0.0, 1.0)] * dims)
    blk.CopyToSeedBuffer(seeds)
    blk.SetNevents(n)
    blk.SubmitKernel(nper=nper, max_tries=tries)
    assert np.array_equal(blk.output.download(), want)
    with pytest.raises(MFError):
        blk.SubmitKernel(nper=nper, max_tries=tries - 1)
    blk.SubmitKernel(nper=nper)
    assert np.array_equal(blk.output.download(), want)
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("workload,n,streams", [("mass", 200003, 8192), ("pwave", 400009, 8192), ("pwave", 6001, 64)])
def test_long_streams_equal_the_streams(workload, n, streams):
    """The models' densities at 8, 16 and 32 lanes of 8 proposals."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import generate_events, generate_partition
    from oracle import mforacle
    b = CUDABackend(0)
    cols = generate_events(b, load_spec(workload), n, seed=mforacle.SEED, max_workitems=streams)
    nper, nseeds = generate_partition(n, streams)
    assert nper >= 24
    assert np.array_equal(cols.download(), mforacle.generate_partitioned(workload, n, nper, nseeds))
    b.close()
