"""The first evaluation of a dataset, which prepares its columns as it reads
them: other block sizes, and columns mapped from the host."""
import numpy as np
import pytest

from morefit_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("workload", ["mass", "pwave"])
@pytest.mark.parametrize("block", [64, 128, 512])
@pytest.mark.parametrize("n", [1, 513, 100003])
def test_first_evaluation_in_other_blocks(workload, block, n):
    """Equal, bit for bit, to the evaluation after it, and so is the copy that
    it leaves (the Hessian's sums after a preparation in a pass of its own)."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import Likelihood, generate_events, load_spec
    b = CUDABackend(0, resident_idle_us=0)
    spec = load_spec(workload)
    theta = np.array(spec["truth"])
    like = Likelihood(b, spec, block=block)
    like.set_device_data(generate_events(b, spec, n, seed=5))
    hess = like.sums("lh_hessian_kernel", theta)
    for kernel in ("lh_kernel", "lh_grad_kernel"):
        want = like.sums(kernel, theta)
        L.lib.mf_buffer_mark_modified(like.input_block(kernel).buf)
        assert np.array_equal(like.sums(kernel, theta), want), kernel
        assert np.array_equal(like.sums(kernel, theta), want), kernel
        assert np.array_equal(like.sums("lh_hessian_kernel", theta), hess), kernel
    b.close()


@pytest.mark.parametrize("workload", ["mass", "cbpoly", "pwave"])
@pytest.mark.parametrize("n", [2, 512, 30010, 200002])
def test_first_evaluation_of_mapped_columns(workload, n):
    """The sums of the same events uploaded, twice (the second mapping of the
    buffer is read anew)."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import Likelihood, generate_events, load_spec
    b = CUDABackend(0, resident_idle_us=0)
    spec = load_spec(workload)
    theta = np.array(spec["truth"])
    host = np.ascontiguousarray(generate_events(b, spec, n, seed=9).download())
    up, mapped = Likelihood(b, spec), Likelihood(b, spec)
    for _ in range(2):
        up.set_data(host)
        mapped.set_data_mapped(host)
        for kernel in ("lh_grad_kernel", "lh_kernel", "lh_grad_kernel"):
            assert np.array_equal(mapped.sums(kernel, theta), up.sums(kernel, theta)), kernel
        b.synchronize()
        host[:] = host[:, ::-1].copy()
    b.close()
