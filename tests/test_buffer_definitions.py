"""Parameter buffers that the gradient and the Hessian both define, in the
kernel that holds both: long texts, callers deep in their stack, FP32."""
import sys

import numpy as np
import pytest

from morefit_gb300 import workloads
from morefit_gb300.workloads import _combined_buffers, _definition, load_spec


def _long(terms):
    return "(" + "+".join(f"({1.0 + i / 7:.15e}*a)" for i in range(terms)) + ")"


@pytest.mark.parametrize("terms", [10, 900, 1000, 5000])
def test_long_definitions_compare(terms):
    assert _definition(_long(terms)) == _definition(_long(terms))
    assert _definition(_long(terms)) != _definition(_long(terms + 1))


def test_definitions_compare_deep_in_the_stack():
    """From a stack with room for 20 more calls: no error, the text stands for itself."""
    text = "(" * 40 + "a" + "+b)" * 40

    def down(n):
        return down(n - 1) if n else _definition(text)
    depth, f = 0, sys._getframe()
    while f:
        depth, f = depth + 1, f.f_back
    assert down(sys.getrecursionlimit() - depth - 20) == text


@pytest.mark.parametrize("workload,shared", [("mass", 11), ("mass_w", 11), ("pwave", 1), ("cbpoly", 24), ("spwave", 14)])
def test_models_share_their_buffers(workload, shared):
    s = load_spec(workload)
    names, added = _combined_buffers(s["grad_buffers"], s["hessian_buffers"], True)
    gname = {n for n, _ in s["grad_buffers"]}
    assert sum(v in gname for v in names.values()) == shared
    assert len(added) == len(s["hessian_buffers"]) - shared


def test_fp32_texts_are_not_compared(monkeypatch):
    monkeypatch.setattr(workloads, "_definition", None)
    s = load_spec("spwave")
    names, added = _combined_buffers(s["grad_buffers"], s["hessian_buffers"], False)
    assert len(set(names.values())) == len(added) == len(s["hessian_buffers"])


@pytest.mark.gpu
@pytest.mark.parametrize("elem", [np.float64, np.float32], ids=["f64", "f32"])
def test_model_with_a_long_buffer_evaluates(elem):
    """A buffer of 5000 terms beside the mass model's own, in value, gradient
    and Hessian: the combined kernel equals the two kernels."""
    import copy
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import Likelihood, generate_events
    b = CUDABackend(0)
    spec = copy.deepcopy(load_spec("mass"))
    events = generate_events(b, spec, 5000, seed=3)
    for buffers, kernel in (("grad_buffers", "lh_grad_kernel"), ("hessian_buffers", "lh_hessian_kernel")):
        name = f"morefit_parambuffer_{len(spec[buffers])}"
        spec[buffers] = list(spec[buffers]) + [(name, _long(5000).replace("*a", f"*{spec['parameters'][0]}"))]
        k = next(k for k in spec["kernels"] if k["name"] == kernel)
        k["params"] = list(k["params"]) + [name]
        k["exprs"] = [f"({e}+({name}*1e-9))" for e in k["exprs"]]
    like = Likelihood(b, spec, elem)
    like.set_device_data(events)
    theta = np.array(spec["truth"])
    f, g, h = like.value_gradient_hessian(theta)
    f1, g1 = like.likelihood_and_gradient(theta)
    tol = 1e-10 if elem == np.float64 else 1e-4
    assert abs(f - f1) <= tol * abs(f1)
    assert np.allclose(g, g1, rtol=tol, atol=tol * abs(f1)) and np.allclose(h, like.hessian(theta), rtol=tol, atol=tol * abs(h).max())
    b.close()
