"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values:

  kind   value      -2 ln L of one dataset            (Likelihood.likelihood)
         gradient   -2 ln L and its gradient          (Likelihood.likelihood_and_gradient)
         hessian    second derivatives                (Likelihood.hessian)
         newton     value, gradient and Hessian       (Likelihood.value_gradient_hessian)
         scan       sums at many parameter points     (Likelihood.sums_many)
         covariance corrected covariance of a weighted fit (Likelihood.corrected_covariance)
         newdata    a new event block on the device: precompute, then value and gradient
         generate   seeded accept-reject events       (generate_events)
         toys       a toy study: generation and fits  (ToyStudy.toy)
  model  a model spec of morefit_gb300/specs
  type   f64 (double) or f32 (mixed precision)
  events events of a dataset (toys: mean events per toy)
  count  parameter points of a scan, toys of a study

The datasets are drawn from the models' own densities, as toy datasets are,
and evaluated a little away from the point they were drawn at, as a fit does.
"""
import json
import math
import os

import numpy as np
import torch

from morefit_gb300 import _lib
from morefit_gb300.backend import CUDABackend, DeviceColumns
from morefit_gb300.toystudy import SegmentSchedule, ToyStudy
from morefit_gb300.workloads import Likelihood, generate_events, load_spec

SPECS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "morefit_gb300", "specs")

# Where datasets are drawn: the models' truth, with the angular asymmetries
# halved so that the density stays positive over the whole angular space
# around it (at the configured truth it is negative in a small corner).
DRAWN_AT = {
    "mass": [5280.0, 20.0, 0.3, -0.002],
    "mass_w": [5280.0, 20.0, 0.3, -0.002],
    "cbpoly": [0.1, 0.05, 1.5, 3.0, -0.3, 0.1, 0.3],
    "pwave": [0.6, -0.005, -0.07, -0.1, -0.05, 0.0, 0.0, 0.0],
    "spwave": [0.6, -0.005, -0.07, -0.1, -0.05, 0.0, 0.0, 0.0, 0.08, -0.05, -0.015, 0.02, 0.01, -0.005],
}
# How far from there they are evaluated (uniform, each parameter).
AWAY = {
    "mass": [1.0, 0.5, 0.01, 1e-4],
    "mass_w": [1.0, 0.5, 0.01, 1e-4],
    "cbpoly": [2e-3, 1e-3, 0.03, 0.1, 0.02, 0.02, 0.01],
    "pwave": [0.01] + [0.008] * 7,
    "spwave": [0.01] + [0.005] * 7 + [0.01] + [0.005] * 5,
}
# Bytes an event takes in the columns an evaluation cannot do without (the
# angular models' linearly independent basis columns, the others' observables).
COLUMNS = {"mass": 1, "mass_w": 2, "cbpoly": 1, "pwave": 9, "spwave": 15}
# Arithmetic an event cannot do without, by output set (a transcendental as 20).
VALUE_OPS = {"mass": 50, "mass_w": 51, "cbpoly": 60, "pwave": 18, "spwave": 30}
NPAR = {"mass": 4, "mass_w": 4, "cbpoly": 7, "pwave": 8, "spwave": 14}
DIMS = {"mass": 1, "mass_w": 2, "cbpoly": 1, "pwave": 3, "spwave": 3}


def listed():
    def case(name, kind, model, type_, events, count=1):
        return {"name": name, "kind": kind, "model": model, "type": type_, "events": events, "count": count}

    return [
        # a fit of a small dataset: every MIGRAD step is one such call
        case("gradient_mass_1k", "gradient", "mass", "f64", 1000),
        # a line-search value of a mixed-precision fit, ragged size
        case("value_pwave_f32_30011", "value", "pwave", "f32", 30011),
        # the headline evaluation: K*mumu P-wave, one million events
        case("gradient_pwave_1M", "gradient", "pwave", "f64", 1000000),
        # the largest dataset, mixed precision: S+P wave with acceptance
        case("gradient_spwave_f32_10M", "gradient", "spwave", "f32", 10000000),
        # HESSE of the headline fit
        case("hessian_pwave_1M", "hessian", "pwave", "f64", 1000000),
        # HESSE of the largest model (105 second derivatives), odd size
        case("hessian_spwave_333333", "hessian", "spwave", "f64", 333333),
        # a Newton step of a fit with conditionals, powers and exponentials
        case("newton_cbpoly_250k", "newton", "cbpoly", "f64", 250000),
        # a likelihood scan: many points of one dataset in one call
        case("scan_pwave_100k_x64", "scan", "pwave", "f64", 100000, 64),
        # the error matrix of a weighted fit
        case("covariance_mass_w_200003", "covariance", "mass_w", "f64", 200003),
        # a fresh dataset: hoisted columns, then the fit's first evaluation
        case("newdata_pwave_1M", "newdata", "pwave", "f64", 1000000),
        # a pseudo-dataset of the headline size
        case("generate_pwave_1M", "generate", "pwave", "f64", 1000000),
        # a toy study: every toy generated at its own truth and fitted
        case("toys_pwave_1000x2000", "toys", "pwave", "f64", 2000, 1000),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["value", "gradient", "gradient", "hessian", "newton", "scan", "covariance", "newdata",
                       "generate", "toys"])
    type_, count = "f64", 1
    if kind in ("value", "gradient"):
        model = rng.choice(["mass", "pwave", "spwave", "cbpoly"])
        type_ = rng.choice(["f64", "f32"])
        events = _log_int(rng, 200, {"spwave": 10000000 if type_ == "f32" else 2000000}.get(model, 4000000))
    elif kind == "hessian":
        model = rng.choice(["mass", "pwave", "spwave", "cbpoly"])
        events = _log_int(rng, 500, 400000 if model == "spwave" else 1000000)
    elif kind == "newton":
        model = rng.choice(["mass", "pwave", "cbpoly"])
        events = _log_int(rng, 500, 400000)
    elif kind == "scan":
        model = rng.choice(["mass", "pwave"])
        count = _log_int(rng, 2, 128)
        events = _log_int(rng, 500, 200000)
    elif kind == "covariance":
        model, events = "mass_w", _log_int(rng, 500, 1000000)
    elif kind == "newdata":
        model = rng.choice(["pwave", "pwave", "spwave"])
        type_ = rng.choice(["f64", "f32"])
        events = _log_int(rng, 500, 1000000)
    elif kind == "generate":
        model = rng.choice(["pwave", "mass", "spwave", "cbpoly"])
        events = _log_int(rng, 500, 1000000 if model == "pwave" else 300000)
    else:
        model, count, events = "pwave", _log_int(rng, 32, 1000), _log_int(rng, 400, 2000)
    return {"kind": kind, "model": model, "type": type_, "events": events, "count": count}


# ------------------------------------------- the models' text, in 64 bits --
def _python(text):
    """The C conditionals of a kernel expression, (c ? a : b), as calls."""
    stack, out = [], ""
    for ch in text:
        if ch == "(":
            stack.append((out, []))
            out = ""
        elif ch in "?:":
            stack[-1][1].append(out)
            out = ""
        elif ch == ")":
            before, parts = stack.pop()
            out = before + ("where(lambda: %s, lambda: %s, lambda: %s)" % (parts[0], parts[1], out) if parts
                            else "(" + out + ")")
        else:
            out += ch
    return out


def _scalar_where(c, a, b):
    return a() if c() else b()


def _tensor_where(c, a, b):
    c = c()
    if not isinstance(c, torch.Tensor):
        return a() if c else b()
    a, b = (v if isinstance(v, torch.Tensor) else torch.full_like(c, v, dtype=torch.float64) for v in (a(), b()))
    return torch.where(c, a, b)


def _either(name):
    s, t = getattr(math, name), getattr(torch, name)
    return lambda x: t(x) if isinstance(x, torch.Tensor) else s(x)


_NAMES = {n: _either(n) for n in ("exp", "log", "sqrt", "sin", "cos", "erf")}


def _evaluate(text, values):
    tensors = any(isinstance(v, torch.Tensor) for v in values.values())
    names = dict(_NAMES, pow=lambda a, b: a ** b, where=_tensor_where if tensors else _scalar_where, **values)
    return eval(compile(_python(text), "<expression>", "eval"), names)


def _spec_text(model):
    with open(os.path.join(SPECS, model + ".json")) as f:
        return json.load(f)


def _kernel_values(spec, kernel, theta, events):
    """Every output of one of the spec's kernels for every event, one at a time."""
    k = next(k for k in spec["kernels"] if k["name"] == kernel)
    buffers = spec[{"lh_kernel": "lh_buffers", "lh_grad_kernel": "grad_buffers",
                    "lh_hessian_kernel": "hessian_buffers", "lh_fisher_kernel": "fisher_buffers"}[kernel]]
    values = dict(zip(spec["parameters"], map(float, theta)))
    for name, text in buffers:
        values[name] = float(_evaluate(text, values))
    raw = dict(zip(spec["dimensions"], events))
    values.update(raw)
    for name, text in spec["event_buffers"]:
        if name != text:
            values[name] = _evaluate(text, raw)
    for text in k["exprs"]:
        yield _evaluate(text, values)


def _sums(spec, kernel, theta, events):
    return np.array([float(v.sum()) for v in _kernel_values(spec, kernel, theta, events)])


def _matrix(sums, npar):
    h = np.zeros((npar, npar))
    i, j = np.tril_indices(npar)
    h[i, j] = h[j, i] = -2.0 * sums
    return h


# ----------------------------------------------------------------- inputs --
def _events(model, n, seed):
    """n events of the model's density at DRAWN_AT: (dimensions, n), on the GPU."""
    source = "mass" if model == "mass_w" else model
    spec = _spec_text(source)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)
    lo, hi = zip(*spec["ranges"])
    bound = 1.1 * next(k for k in spec["kernels"] if k.get("generate"))["maxprob"]
    kept, have = [], 0
    while have < n:
        u = torch.rand((len(lo) + 1, min(1 << 22, 1024 + 12 * (n - have))), generator=gen, device="cuda",
                       dtype=torch.float64)
        x = torch.stack([a + (b - a) * u[d] for d, (a, b) in enumerate(zip(lo, hi))])
        log_p = next(_kernel_values(spec, "lh_kernel", DRAWN_AT[model], list(x)))
        x = x[:, bound * u[-1] < torch.exp(log_p)]
        kept.append(x)
        have += x.shape[1]
    x = torch.cat(kept, dim=1)[:, :n]
    if model == "mass_w":  # weights in [0.5, 1.5), as an efficiency correction has them
        x = torch.cat([x, 0.5 + torch.rand((1, n), generator=gen, device="cuda", dtype=torch.float64)])
    return x.contiguous()


def _points(model, seed, count):
    u = np.random.default_rng(int(seed) + 101).uniform(-1.0, 1.0, (count, NPAR[model]))
    return np.array(DRAWN_AT[model]) + u * np.array(AWAY[model])


_backend = None


def _the_backend():
    """One backend for the program, as its datasets and kernels share it."""
    global _backend
    if _backend is None:
        _backend = CUDABackend(0)
    return _backend


class _Block:
    """A device event block as a tensor (columns at their stride), kept alive with it."""

    def __init__(self, cols):
        self.cols = cols
        self.__cuda_array_interface__ = {
            "shape": (cols.ncols, cols.n), "strides": (cols.stride * cols.itemsize, cols.itemsize),
            "typestr": "<f8" if cols.itemsize == 8 else "<f4", "version": 3,
            "data": (int(_lib.lib.mf_buffer_device_ptr(cols.buf)), False)}


def prepare(case, seed):
    backend, model, n = _the_backend(), case["model"], case["events"]
    spec = load_spec(model)
    state = {"case": case, "spec": spec, "seed": int(seed)}
    if case["kind"] == "generate":
        return state
    if case["kind"] == "toys":
        # the schedule that a study of this size settles on
        state["study"] = ToyStudy(backend, spec, seed=int(seed), schedule=SegmentSchedule(128, 0))
        return state
    kernel_type = np.float32 if case["type"] == "f32" else np.float64
    state["like"] = Likelihood(backend, spec, kernel_type)
    state["points"] = _points(model, seed, case["count"])
    events = _events(model, n, seed).cpu().numpy()
    if case["kind"] == "newdata":
        state["columns"] = DeviceColumns(backend, state["like"].pre.elem)
        state["columns"].upload(events)
    else:
        state["like"].set_data(events)
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "generate":
        cols = generate_events(_the_backend(), state["spec"], case["events"], seed=state["seed"])
        return torch.as_tensor(_Block(cols), device="cuda")
    if kind == "toys":
        r = state["study"].toy(case["count"], case["events"], poisson=True, clip=(200, 50000), jitter=0.1)
        return {"values": r.fit.values, "errors": r.fit.errors, "fmin": r.fit.fmin, "pulls": r.pulls,
                "truth": r.truth, "counts": r.counts, "converged": r.fit.converged}
    like, theta = state["like"], state["points"][0]
    if kind == "value":
        return like.likelihood(theta)
    if kind == "gradient":
        return like.likelihood_and_gradient(theta)
    if kind == "hessian":
        return like.hessian(theta)
    if kind == "newton":
        return like.value_gradient_hessian(theta)
    if kind == "scan":
        return like.sums_many("lh_grad_kernel", state["points"])
    if kind == "covariance":
        return like.corrected_covariance(theta)
    like.set_device_data(state["columns"])
    return like.likelihood_and_gradient(theta)


def work(case):
    model, kind, n, count = case["model"], case["kind"], case["events"], case["count"]
    size = 4 if case["type"] == "f32" else 8
    npar = NPAR[model]
    nhess = npar * (npar + 1) // 2
    value = VALUE_OPS[model]
    gradient, hessian = value + 4 * npar, value + 4 * npar + 2 * nhess
    if kind == "generate":
        # every accepted event: its coordinates written and one density
        return {"bytes": 8.0 * DIMS[model] * n, "flops": float(n * (value + 60))}
    if kind == "toys":
        # the events of every toy written once and read once, one Newton step
        return {"bytes": 2.0 * 8 * 3 * n * count, "flops": float(n * count * (hessian + 60))}
    flops = {"value": value, "gradient": gradient, "hessian": hessian, "newton": hessian, "scan": gradient,
             "covariance": hessian + 2 * nhess, "newdata": gradient + 150}[kind]
    if kind == "newdata":
        return {"bytes": float(size * n * DIMS[model]), "flops": float(flops * n)}
    if case["type"] == "f32" and model in ("mass", "cbpoly"):
        size = 8  # raw observables keep their FP64 storage
    return {"bytes": float(size * n * COLUMNS[model]), "flops": float(flops * n * count)}


# ------------------------------------------------------------------ exact --
def _bits(words):
    """(rows, 4) 32-bit words as (rows, 128) bits, least significant first."""
    return np.unpackbits(np.ascontiguousarray(words.astype("<u4")).view(np.uint8), axis=1, bitorder="little")


def _words(bits):
    return np.packbits(bits, axis=1, bitorder="little").view("<u4").astype(np.uint32)


def _next(s):
    """xoshiro128++ over rows of states, in place; its outputs."""
    rotl = lambda x, k: (x << np.uint32(k)) | (x >> np.uint32(32 - k))  # noqa: E731
    r = rotl(s[0] + s[3], 7) + s[0]
    t = s[1] << np.uint32(9)
    s[2] ^= s[0]
    s[3] ^= s[1]
    s[1] ^= s[2]
    s[0] ^= s[3]
    s[2] ^= t
    s[3] = rotl(s[3], 11)
    return r


def _streams(seed, rows):
    """xoshiro128++ states: SplitMix64 of the seed, then one jump() a row (a
    linear map of the 128 state bits, applied by doubling)."""
    z, first = int(seed), []
    for _ in range(4):
        z = (z + 0x9E3779B97F4A7C15) & (2**64 - 1)
        y = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & (2**64 - 1)
        y = ((y ^ (y >> 27)) * 0x94D049BB133111EB) & (2**64 - 1)
        first.append((y ^ (y >> 31)) >> 32)
    s = np.ascontiguousarray(_words(np.eye(128, dtype=np.uint8)).T)
    total = np.zeros_like(s)
    for word in (0x8764000B, 0xF542D2D3, 0x6FA035C3, 0x77F2DB5B):
        for bit in range(32):
            if word >> bit & 1:
                total ^= s
            _next(s)
    jump = _bits(total.T).astype(np.int64)  # row i: the image of state bit i
    states = _bits(np.array([first], dtype=np.uint32))
    while len(states) < rows:
        states = np.concatenate([states, (states.astype(np.int64) @ jump & 1).astype(np.uint8)])
        jump = jump @ jump & 1
    return np.ascontiguousarray(_words(states[:rows]).T)


def _exact_generate(case, seed):
    """The seeded accept-reject events: one stream a generator thread (the
    reference's partition, at most 8192 threads)."""
    spec, n = _spec_text(case["model"]), case["events"]
    gen = next(k for k in spec["kernels"] if k.get("generate"))
    per = n // 8192 + 1 if n > 8192 else 1
    s = _streams(seed, -(-n // per))
    printed = lambda v: float("%.15e" % v)  # noqa: E731
    begin = np.arange(s.shape[1], dtype=np.int64) * per
    end, at = np.minimum(begin + per, n), begin.copy()
    out = np.empty((len(gen["lo"]), n))
    while (at < end).any():
        u = [_next(s) * 2.3283064365386963e-10 for _ in range(len(gen["lo"]) + 1)]
        x = [printed(a) + printed(b - a) * v for a, b, v in zip(gen["lo"], gen["hi"], u)]
        p = _evaluate(gen["exprs"][0], {d: torch.from_numpy(v) for d, v in zip(gen["outputs"], x)}).numpy()
        take = np.nonzero((printed(gen["maxprob"]) * u[-1] < p) & (at < end))[0]
        for d, v in enumerate(x):
            out[d, at[take]] = v[take]
        at[take] += 1
    return out


def exact(case, seed):
    kind, model = case["kind"], case["model"]
    if kind == "toys":
        return None  # a fit ends where its own stopping rule ends it
    if kind == "generate":
        return _exact_generate(case, seed)
    spec = _spec_text(model)
    events = list(_events(model, case["events"], seed))
    points = _points(model, seed, case["count"])
    theta, npar = points[0], NPAR[model]
    if kind == "value":
        return -2.0 * _sums(spec, "lh_kernel", theta, events)[0]
    if kind == "scan":
        return np.array([_sums(spec, "lh_grad_kernel", t, events) for t in points])
    if kind in ("hessian", "covariance"):
        h = _matrix(_sums(spec, "lh_hessian_kernel", theta, events), npar)
        if kind == "hessian":
            return h
        f = _matrix(_sums(spec, "lh_fisher_kernel", theta, events), npar)
        hinv = np.linalg.inv(h)
        return -2.0 * hinv @ f @ hinv
    s = _sums(spec, "lh_grad_kernel", theta, events)
    if kind == "newton":
        h = _matrix(_sums(spec, "lh_hessian_kernel", theta, events), npar)
        return float(-2.0 * s[0]), -2.0 * s[1:], h
    return float(-2.0 * s[0]), -2.0 * s[1:]
