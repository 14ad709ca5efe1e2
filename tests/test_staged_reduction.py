"""Block reduction of FP32 kernels of few outputs: a warp per output through
shared memory, within 16 KB of it."""
import numpy as np
import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import compile_check, lower_source


def _exprs(outputs):
    return [f"exp((x*a*{j}.25))" for j in range(outputs)]


@pytest.mark.parametrize("outputs,block,staged", [(1, 256, True), (5, 256, True), (8, 256, True), (9, 256, False),
                                                  (2, 64, True), (3, 64, False), (2, 1024, True), (3, 1024, False),
                                                  (4, 512, True), (5, 512, False)])
def test_which_kernels_stage(outputs, block, staged):
    args = ("k", L.MF_KERNEL_REDUCE, L.MF_F32, ["x"], ["a"], _exprs(outputs))
    assert ("mf_stage[MF_NOUT]" in lower_source(*args, block=block)) == staged
    if staged:
        assert compile_check(*args, block=block)["spill_bytes"] == 0
    for native in (False, True):
        assert "mf_stage[" not in lower_source("k", L.MF_KERNEL_REDUCE, L.MF_F64, *args[3:], block=block, native_f64=native)


@pytest.mark.gpu
@pytest.mark.parametrize("outputs,block", [(1, 256), (5, 256), (8, 256), (9, 256), (2, 64), (2, 1024), (4, 512), (1, 96)])
@pytest.mark.parametrize("n", [1, 257, 70001])
def test_staged_sums_match_fp64(outputs, block, n):
    """Single and segment sums."""
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0, resident_idle_us=0)
    x = np.random.default_rng(n).uniform(-1.0, 1.0, n).astype(np.float32)
    blk = CUDABlock(b, np.float32, block=block)
    blk.MakeComputeKernel("k", 0, ["x"], ["r"] * outputs, ["a"], _exprs(outputs), True)
    blk.CopyToInputBuffer(x[None, :])
    blk.CopyToParameterBuffer([0.5])
    blk.SubmitKernel()
    ref = np.array([np.exp(x.astype(np.float64) * 0.5 * (j + 0.25)).sum() for j in range(outputs)])
    # positive terms: a few FP32 roundings of the argument and the function
    tol = 2.0**-19
    assert (np.abs(blk.CopyFromKahanBuffer() - ref) <= tol * ref).all()
    seg = blk.SubmitSegments([0, 0], [n, max(1, n // 3)], [[0.5], [0.5]])
    assert (np.abs(seg[0] - ref) <= tol * ref).all()
    b.close()
