"""Segments without events, parameters that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e39])
@pytest.mark.parametrize("events_per_block", [0, 256])
def test_empty_segments_sum_to_zero_at_once(value, events_per_block):
    """Outputs with a parameter-only factor, which is applied to the sum: zero
    for an empty segment whatever the factor, without a second evaluation in
    native FP64; the segment beside it as alone."""
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0)
    blk = CUDABlock(b, np.float64)
    blk.MakeComputeKernel("empty", 0, ["x"], ["r"] * 2, ["a"], ["(x*a)", "((x*x)*a)"], True)
    blk.CopyToInputBuffer(np.linspace(0.5, 2.0, 300)[None, :])
    got = blk.SubmitSegments([0, 0, 300], [0, 300, 0], [[value], [1.5], [value]], events_per_block)
    assert np.array_equal(got[[0, 2]], np.zeros((2, 2)))
    assert np.array_equal(got[1], blk.SubmitSegments([0], [300], [[1.5]], events_per_block)[0])
    assert blk.kernel.fallback_count() == 0
    b.close()
