"""The first evaluation of a dataset, which prepares its columns as it reads
them: the sums, and the prepared copy that it leaves, bit for bit those of the
preparation in a pass of its own."""
import numpy as np
import pytest

from morefit_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _reduce(like, kernel, cols, n, theta):
    k = like.blocks[kernel].kernel
    row = np.ascontiguousarray(like.param_rows(kernel, theta[None]))[0]
    out = np.empty(k.nout)
    L.check(L.lib.mf_kernel_reduce(k.handle, cols.buf, cols.stride, n, L.dptr(row), row.size, L.dptr(out)))
    return out


@pytest.mark.parametrize("workload", ["mass", "pwave"])
@pytest.mark.parametrize("kernel", ["lh_kernel", "lh_grad_kernel"])
@pytest.mark.parametrize("n", [1, 2, 511, 513, 155649, 200001])
def test_first_evaluation_equals_the_prepared_ones(workload, kernel, n):
    """Odd and ragged sizes, less and more than one turn of the grid, every
    event and (the columns' other rows prepared too) a part of them first."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import Likelihood, generate_events, load_spec
    b = CUDABackend(0, resident_idle_us=0)
    spec = load_spec(workload)
    theta = np.array(spec["truth"])
    events = generate_events(b, spec, n, seed=5)
    ref = Likelihood(b, spec)
    ref.set_device_data(events)
    hess = ref.sums("lh_hessian_kernel", theta)  # its columns prepared in a pass of their own
    want = ref.sums(kernel, theta)
    like = Likelihood(b, spec)
    for part in (n, n - n // 9, max(1, n // 2)):
        like.set_device_data(events)
        cols = like.input_block(kernel)
        L.lib.mf_buffer_mark_modified(cols.buf)
        first = _reduce(like, kernel, cols, part, theta)
        assert np.array_equal(like.sums(kernel, theta), want), part
        assert np.array_equal(like.sums("lh_hessian_kernel", theta), hess), part
        assert np.array_equal(_reduce(like, kernel, cols, part, theta), first), part
        if part == n:
            assert np.array_equal(first, want)
    b.close()
