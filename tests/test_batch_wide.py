"""Batches of evaluations of many columns on either side of the rule that sends
them to one launch or to a launch each."""
import ctypes as C

import numpy as np
import pytest

from test_prefetch_fits import value_and_gradient

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [25, 48, 64])
@pytest.mark.parametrize("n", [1, 8000, 15000, 16000, 24000, 39000, 40000])
def test_batched_equal_single(columns, n):
    from morefit_gb300 import _lib as L
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0, resident_idle_us=0)
    cols, exprs = value_and_gradient(columns, 3)
    blk = CUDABlock(b, np.float64)
    blk.MakeComputeKernel("k", 0, cols, ["r"] * 3, [f"a{i}" for i in range(4)], exprs, True)
    blk.CopyToInputBuffer(np.random.default_rng(n).uniform(0.5, 1.5, (columns, n)))
    count = 9
    rows = np.random.default_rng(1).uniform(0.1, 0.4, (count, 4))
    out = L.c_buf()
    L.check(L.lib.mf_buffer_alloc(b.handle, count * 3 * 8, C.byref(out)))
    u64p = C.POINTER(C.c_uint64)
    st, ns = np.full(count, blk.input.stride, np.uint64), np.full(count, n, np.uint64)
    L.check(L.lib.mf_kernel_reduce_many(blk.kernel.handle, count, (L.c_buf * count)(*([blk.input.buf] * count)),
                                        st.ctypes.data_as(u64p), ns.ctypes.data_as(u64p), L.dptr(rows), 4, out))
    got = np.empty((count, 3))
    L.check(L.lib.mf_buffer_d2h(out, 0, got.ctypes.data, got.nbytes))
    L.lib.mf_buffer_free(out)
    for i in range(count):
        blk.CopyToParameterBuffer(rows[i])
        blk.SubmitKernel()
        assert np.array_equal(blk.CopyFromKahanBuffer(), got[i]), i
    b.close()
