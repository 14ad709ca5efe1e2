"""Register spills of Hessians of many parameters (CPU: NVRTC for sm_103a)."""
import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import compile_check


def hessian(p):
    """The Hessian of a sum of logarithms of a density linear in p + 1 columns."""
    den = "c0"
    for i in range(p):
        den = f"({den}+(t{i}*c{i + 1}))"
    return ([f"c{i}" for i in range(p + 1)], [f"t{i}" for i in range(p)],
            [f"(-(c{i + 1}*c{j + 1})*1.0/(({den}*{den})))" for i in range(p) for j in range(i + 1)])


# spilled bytes a thread: none where the partials fit beside the event loop,
# else what the loop's own partials beyond the registers take (and a few
# bytes of the allocator's choice)
@pytest.mark.parametrize("p,limit", [(14, 0), (15, 0), (16, 0), (18, 600), (20, 1350)])
def test_hessian_reduction_adds_no_spill(p, limit):
    cols, params, exprs = hessian(p)
    r = compile_check("h", L.MF_KERNEL_REDUCE, L.MF_F64, cols, params, exprs)
    assert r["spill_bytes"] <= limit, r
