"""Many small evaluations in one launch (mf_kernel_reduce_many below one grid
of the device): every row equals the evaluation's own launch bit for bit."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_golden

pytestmark = pytest.mark.gpu


def _many(like, kernel, blocks, thetas):
    """reduce_many over datasets `blocks` (DeviceColumns), one parameter point each."""
    from morefit_gb300 import _lib as L
    k = like.blocks[kernel].kernel
    rows = np.ascontiguousarray(like.param_rows(kernel, thetas))
    count = len(blocks)
    out = L.c_buf()
    L.check(L.lib.mf_buffer_alloc(like.backend.handle, count * k.nout * 8, C.byref(out)))
    u64p = C.POINTER(C.c_uint64)
    ins = (L.c_buf * count)(*[b.buf for b in blocks])
    strides = np.array([b.stride for b in blocks], dtype=np.uint64)
    ns = np.array([b.n for b in blocks], dtype=np.uint64)
    L.check(L.lib.mf_kernel_reduce_many(k.handle, count, ins, strides.ctypes.data_as(u64p), ns.ctypes.data_as(u64p),
                                        L.dptr(rows), rows.shape[1], out))
    res = np.empty((count, k.nout))
    L.check(L.lib.mf_buffer_d2h(out, 0, res.ctypes.data, res.nbytes))
    L.lib.mf_buffer_free(out)
    return res


@pytest.mark.parametrize("workload", ["mass", "pwave"])
@pytest.mark.parametrize("kernel", ["lh_kernel", "lh_grad_kernel"])
@pytest.mark.parametrize("count", [2, 9, 64, 65, 130])
def test_points_of_one_dataset(workload, kernel, count):
    """One to three launches of points, groups of one and of several a block."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import Likelihood, generate_events
    g = load_golden(f"{workload}_n1000.json")
    b = CUDABackend(0, resident_idle_us=0)
    truth = np.array(g["truth"])
    for n in (1, 511, 513, 30011, 70001):
        like = Likelihood(b, g)
        like.set_device_data(generate_events(b, g, n, seed=n))
        th = truth * (1.0 + 1e-3 * np.sin(np.arange(truth.size)[None, :] + np.arange(count)[:, None]))
        many = like.sums_many(kernel, th)
        for i in {0, 1, count // 2, count - 1}:
            assert np.array_equal(many[i], like.sums(kernel, th[i])), (n, i)
    b.close()


def test_datasets_of_several_sizes():
    """Datasets that change within a block's group, sizes from one event to the
    largest that leaves the device a block short, and one beyond it (which sends
    the whole batch to a launch each)."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import Likelihood, generate_events
    g = load_golden("pwave_n1000.json")
    b = CUDABackend(0, resident_idle_us=0)
    sms = b.properties()["sms"]
    truth = np.array(g["truth"])
    like = Likelihood(b, g)
    sizes = [1, 30, 512, 513, 5000, (sms - 1) * 512, 77, 5000, 1024, 300 * sms]
    likes = []
    for i, n in enumerate(sizes + [40 * sms * 512]):
        lk = Likelihood(b, g)
        lk.set_device_data(generate_events(b, g, n, seed=100 + i))
        likes.append(lk)
    order = [0, 1, 1, 2, 3, 5, 5, 4, 6, 7, 8, 9, 0, 3, 3, 3, 5, 2]
    for extra in ([], [10]):
        use = order + extra
        th = truth * (1.0 + 1e-3 * np.sin(np.arange(truth.size)[None, :] + np.arange(len(use))[:, None]))
        got = _many(like, "lh_grad_kernel", [likes[i].input_block() for i in use], th)
        for q, i in enumerate(use):
            assert np.array_equal(got[q], likes[i].sums("lh_grad_kernel", th[q])), (q, sizes[i] if i < 10 else "large")
    b.close()


@pytest.mark.parametrize("turns,off", [(1, 0), (1, 1), (2, -1), (2, 0), (2, 1), (3, 0), (3, 1)])
def test_prefetching_loop_reads_the_same_events(turns, off):
    """A lone Hessian, whose loop loads one turn of the grid ahead and asks for
    another in L2, against the batched entry's plain loop, at events around
    whole turns: the same sums bit for bit."""
    from morefit_gb300.backend import CUDABackend
    from morefit_gb300.workloads import Likelihood, generate_events, load_spec
    import torch
    b = CUDABackend(0, resident_idle_us=0)
    n = turns * 256 * torch.cuda.get_device_properties(0).multi_processor_count + off
    like = Likelihood(b, load_spec("pwave"))
    cols = generate_events(b, load_spec("pwave"), n, seed=3)
    like.set_device_data(cols)
    theta = np.array(load_spec("pwave")["truth"])
    lone = like.sums("lh_hessian_kernel", theta)
    many = like.sums_many("lh_hessian_kernel", np.stack([theta, theta]))
    assert np.array_equal(many[0], lone) and np.array_equal(many[1], lone)
    b.close()
