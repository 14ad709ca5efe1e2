"""Kernels built from one description share their loaded code: each runs on
after the other is freed, and a later build loads it again."""
import ctypes as C

import numpy as np
import pytest

from conftest import golden_events, kernel_spec, load_golden

pytestmark = pytest.mark.gpu


def test_kernels_of_one_image_outlive_each_other():
    from morefit_gb300 import _lib as L
    from morefit_gb300.backend import CUDABackend, DeviceColumns, build_kernel
    g = load_golden("mass_n1000.json")
    k = kernel_spec(g, "lh_grad_kernel")
    pt = g["points"][0]
    par = np.ascontiguousarray(pt["kernel_params"]["lh_grad_kernel"])
    backends = [CUDABackend(0, resident_idle_us=0) for _ in range(2)]
    cols = []
    for b in backends:
        c = DeviceColumns(b, L.MF_F64)
        c.upload(golden_events("mass", 1000))
        cols.append(c)

    def make(i):
        return build_kernel(backends[i], "lh_grad_kernel", L.MF_KERNEL_REDUCE, L.MF_F64, k["inputs"], k["params"], k["exprs"])

    def run(i, kern):
        out = np.zeros(kern.nout)
        L.check(L.lib.mf_kernel_reduce(kern.handle, cols[i].buf, cols[i].stride, 1000, L.dptr(par), kern.nparams,
                                       L.dptr(out)))
        return out
    a, b2 = make(0), make(1)
    ref = run(0, a)
    assert np.array_equal(run(1, b2), ref)
    L.check(L.lib.mf_kernel_free(a.handle))
    assert np.array_equal(run(1, b2), ref)
    L.check(L.lib.mf_kernel_free(b2.handle))
    c = make(0)
    assert np.array_equal(run(0, c), ref)
    L.check(L.lib.mf_kernel_free(c.handle))
    for x in cols:
        x.free()
    for x in backends:
        x.close()
