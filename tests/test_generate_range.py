"""FP64 generation with constants and ranges beyond FP32's: the kernels build,
the FP32 accept test's bounds cover what FP32 cannot hold, and the events are
those of one thread walking each stream in FP64."""
import re

import numpy as np
import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import compile_check, lower_source

NEAR_FP32 = float(np.float32(3e-31)) * (1.0 + 2.0**-52)  # 2^-153 from an FP32 number, without being one

# density text, the same in Python, range, bound
CASES = {
    "constant 1e-38": ("((1e-38+x0)*x0)", lambda x: (1e-38 + x) * x, (0.0, 1.0), 1.0),
    "constant 1e-40": ("(1e-40+x0)", lambda x: 1e-40 + x, (0.0, 1.0), 1.0),
    "constant 1e-60": ("(1e-60+x0)", lambda x: 1e-60 + x, (0.0, 1.0), 1.0),
    "constant 1e-300": ("(x0*(x0+1e-300))", lambda x: x * (x + 1e-300), (0.0, 1.0), 1.0),
    "constants that cancel": ("((x0*1e-60)*1e60)", lambda x: x * 1e-60 * 1e60, (0.0, 1.0), 1.0),
    "constant 1e300": ("((x0*1e300)*1e-300)", lambda x: x * 1e300 * 1e-300, (0.0, 1.0), 1.0),
    "constant next to an FP32 number": (f"((x0*{NEAR_FP32!r})*1e31)", lambda x: x * NEAR_FP32 * 1e31, (0.0, 1.0), 3.0),
    "range of 1e-40": ("(x0*1e40)", lambda x: x * 1e40, (0.0, 1e-40), 1.0),
    "range of 1e-50": ("(x0*1e50)", lambda x: x * 1e50, (0.0, 1e-50), 1.0),
    "range of 1e-37": ("(x0*1e37)", lambda x: x * 1e37, (0.0, 1e-37), 1.0),
    "range to 1e39": ("(x0*1e-39)", lambda x: x * 1e-39, (0.0, 1e39), 1.0),
    "range -3e38 ... 3e38": ("((x0*1e-39)*(x0*1e-39))", lambda x: (x * 1e-39) * (x * 1e-39), (-3e38, 3e38), 0.09),
    "bound of 1e-50": ("(x0*1e-50)", lambda x: x * 1e-50, (0.0, 1.0), 1e-50),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_generate_kernel_builds(name):
    text, _, rng, maxprob = CASES[name]
    compile_check("g", L.MF_KERNEL_GENERATE, L.MF_F64, [], [], [text], gen=(["x0"], [rng[0]], [rng[1]], maxprob))


@pytest.mark.parametrize("name", sorted(CASES))
def test_coordinate_and_constant_bounds_hold(name):
    """The FP32 coordinate's distance from the FP64 one and every constant's
    from its own, against the bounds in the source."""
    text, _, (lo, hi), maxprob = CASES[name]
    src = lower_source("g", L.MF_KERNEL_GENERATE, L.MF_F64, [], [], [text], gen=(["x0"], [lo], [hi], maxprob))

    def value(t):
        return np.inf if t == "MF_EF_INF" else float(np.float32(t.strip("()").rstrip("f")))
    m = re.search(r"const mf_ef xe0 = mf_ef_make\((?:__fmaf_rn\((.*), \(float\)d0 \* 2.3283064365386963e-10f, (.*)\)|0.0f), (.*)\);", src)
    bound = value(m.group(3))
    if np.isfinite(bound):
        u = np.concatenate([[0.0, 1.0], np.random.default_rng(1).random(1000)])
        got = (np.float64(value(m.group(1))) * u.astype(np.float32) + value(m.group(2))).astype(np.float32)
        assert (np.abs(got.astype(np.float64) - (lo + (hi - lo) * u)) <= bound).all()
    body = src[src.index("mf_ef mf_filter("):]
    body = body[:body.index("return")]
    made = re.findall(r"mf_ef_make\(([^,()]*|\([^()]*\)), ([^()]*?)\)", body)
    want = {float(c) for c in re.findall(r"\d[\d.]*e[+-]?\d+", text)}
    assert len(made) >= len(want)
    for c in want:
        assert any(abs(value(v) - c) <= value(e) for v, e in made), c


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("nper", [7, 40])
def test_events_equal_the_streams(name, nper):
    from morefit_gb300.backend import CUDABackend, CUDABlock
    from morefit_gb300.workloads import seed_rows
    text, density, (lo, hi), maxprob = CASES[name]
    streams = 50
    n = streams * nper - 3
    seeds = seed_rows(streams, 91)
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
        return r.astype(np.float64) * 2.3283064365386963e-10
    want, got = np.zeros(n), np.zeros(streams, np.int64)
    quota = np.minimum(nper, n - nper * np.arange(streams))
    while (got < quota).any():
        x = lo + (hi - lo) * draw()
        take = (maxprob * draw() < density(x)) & (got < quota)
        want[(nper * np.arange(streams) + got)[take]] = x[take]
        got += take
    b = CUDABackend(0)
    blk = CUDABlock(b, np.float64)
    blk.MakeGenerateKernel("g", n, [], ["x0"], [], [text], maxprob, ranges=[(lo, hi)])
    blk.CopyToSeedBuffer(seeds)
    blk.SetNevents(n)
    blk.SubmitKernel(nper=nper)
    assert np.array_equal(blk.output.download()[0], want)
    b.close()
