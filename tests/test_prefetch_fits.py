"""Entries that load the next events while they compute: not where two vectors
of the columns and the partials exceed the registers (CPU: NVRTC for sm_103a)."""
import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import compile_check, lower_source
from morefit_gb300.workloads import load_spec


def value_and_gradient(columns, outputs):
    cols = [f"c{i}" for i in range(columns)]
    den = "(" + "+".join(["c0"] + [f"(a{i % 4}*c{i + 1})*c{i}" for i in range(columns - 1)]) + ")"
    return cols, [f"log({den})"] + [f"(c{i}*1.0/({den}))" for i in range(outputs - 1)]


# 31 columns and 5 outputs still prefetch: 276 bytes, and faster for it
@pytest.mark.parametrize("columns,outputs,limit", [(25, 1, 0), (31, 1, 0), (31, 5, 300), (37, 1, 0), (37, 5, 0), (48, 1, 0)])
def test_many_columns_do_not_spill(columns, outputs, limit):
    cols, exprs = value_and_gradient(columns, outputs)
    r = compile_check("k", L.MF_KERNEL_REDUCE, L.MF_F64, cols, [f"a{i}" for i in range(4)], exprs)
    assert r["spill_bytes"] <= limit, r


@pytest.mark.parametrize("block", [256, 384, 512])
def test_hessian_in_larger_blocks_does_not_spill(block):
    k = next(k for k in load_spec("pwave")["kernels"] if k["name"] == "lh_hessian_kernel")
    r = compile_check("k", L.MF_KERNEL_REDUCE, L.MF_F64, k["inputs"], k["params"], k["exprs"], block=block)
    assert r["spill_bytes"] == 0, r


@pytest.mark.parametrize("columns,first", [(16, True), (31, True), (37, False), (64, False)])
def test_first_entry_where_it_fits(columns, first):
    cols, exprs = value_and_gradient(columns, 1)
    src = lower_source("k", L.MF_KERNEL_REDUCE, L.MF_F64, cols, [f"a{i}" for i in range(4)], exprs)
    assert ("mf_reduce_first(" in src) == first


@pytest.mark.gpu
@pytest.mark.parametrize("columns", [16, 31, 37, 64])
@pytest.mark.parametrize("n", [1, 513, 77777])
def test_many_columns_match_fp64(columns, n):
    """Single, first, batched and segment sums on either side of the rule."""
    import numpy as np
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0, resident_idle_us=0)
    cols, exprs = value_and_gradient(columns, 5)
    a = np.array([0.1, 0.2, 0.3, 0.4])
    x = np.random.default_rng(n).uniform(0.5, 1.5, (columns, n))
    den = x[0] + sum(a[i % 4] * x[i + 1] * x[i] for i in range(columns - 1))
    ref = np.stack([np.log(den)] + [x[i] / den for i in range(4)]).sum(axis=1)
    blk = CUDABlock(b, np.float64)
    blk.MakeComputeKernel("k", 0, cols, ["r"] * 5, [f"a{i}" for i in range(4)], exprs, True)
    blk.CopyToInputBuffer(x)
    blk.CopyToParameterBuffer(a)
    for _ in range(2):  # the first evaluation prepares the columns
        blk.SubmitKernel()
        # 2^-44 for each of about 2 x columns operations of one event, of either sign over events
        assert np.allclose(blk.CopyFromKahanBuffer(), ref, rtol=2.0**-44 * 2 * columns, atol=0)
    assert np.allclose(blk.SubmitSegments([0], [n], [a])[0], ref, rtol=2.0**-44 * 2 * columns, atol=0)
    b.close()
