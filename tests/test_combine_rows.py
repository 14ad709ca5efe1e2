"""The combine of block rows: one round of loads for a full grid of a kernel of
one output, whose every thread takes rows, and the sums of few outputs at grids
around its edges."""
import math
import re

import numpy as np
import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import lower_source


def _exprs(outputs):
    return ["sqrt(x)"] + [f"(x*a*{j}.5)" for j in range(1, outputs)]


@pytest.mark.parametrize("block", [64, 256, 1024])
@pytest.mark.parametrize("elem", [L.MF_F64, L.MF_F32])
def test_full_grids_of_one_output_combine_in_one_round(block, elem):
    """Up to eight blocks of 256 threads on each of 152 SMs (16 loads a thread are the most)."""
    src = lower_source("k", L.MF_KERNEL_REDUCE, elem, ["x"], ["a"], _exprs(1), block=block)
    grp, q = (int(re.search(rf"#define {m} (\d+)", src).group(1)) for m in ("MF_GRP", "MF_Q"))
    assert grp == block and grp * q >= min(8 * 152, 16 * block)


@pytest.mark.gpu
@pytest.mark.parametrize("elem", [np.float64, np.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("outputs,block", [(1, 256), (2, 256), (3, 256), (5, 256), (7, 256), (8, 256), (9, 256), (1, 64),
                                           (1, 1024), (2, 96)])
def test_sums_at_the_edges_of_the_combine(elem, outputs, block):
    """Grids of 1, 31 to 33 rows, around the rows of one per thread and of full
    rounds, and the largest; single, batched and (first) prepared evaluations
    give one value, within the operations' rounding of the exact sum."""
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0, resident_idle_us=0)
    rng = np.random.default_rng(block + outputs)
    blk = CUDABlock(b, elem, block=block)
    blk.MakeComputeKernel("rows", 0, ["x"], ["r"] * outputs, ["a"], _exprs(outputs), True)
    vec = blk.kernel.info()["vec"]
    grp = block if outputs == 1 else min(32, block // outputs)
    rows = {1, 31, 32, 33, grp - 1, grp, grp + 1, 2 * grp + 1, 16 * grp + 1, 2000}
    for r in sorted(v for v in rows if 1 <= v <= 2000):
        n = r * block * vec - (r * 7) % (block * vec)
        x = rng.uniform(0.5, 1.5, n).astype(elem)
        blk.CopyToInputBuffer(x[None, :])
        blk.CopyToParameterBuffer([0.75])
        blk.SubmitKernel()
        got = blk.CopyFromKahanBuffer()
        blk.SubmitKernel()
        assert np.array_equal(got, blk.CopyFromKahanBuffer()), r
        xd = x.astype(np.float64)
        ref = np.array([math.fsum(np.sqrt(xd))] + [0.75 * (j + 0.5) * math.fsum(xd) for j in range(1, outputs)])
        # FP64: a few double-float operations an event; FP32: a few roundings an event, all of one sign at worst
        tol = 2.0**-42 if elem == np.float64 else 2.0**-21
        assert (np.abs(got - ref) <= tol * np.abs(ref)).all(), (r, got, ref)
    b.close()
