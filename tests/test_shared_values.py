"""Values that several outputs of a kernel share: operands in another order,
powers of one base and its logarithm, a reciprocal and its square, parameter
buffers the gradient and the Hessian both define."""
import numpy as np
import pytest

from morefit_gb300 import _lib as L
from morefit_gb300.backend import lower_source


def _part(src):
    i = src.index("mf_reduce_part(")
    return src[i:src.index('extern "C"', i)]


def test_exchanged_operands_and_powers_share():
    exprs = ["sqrt(((a*x)+y))", "((y+(x*a))*sqrt((y+(a*x))))", "(pow(x,a)+(pow(x,2.5)*log(x)))", "(1.0/(x)+1.0/((x*x)))"]
    part = _part(lower_source("k", L.MF_KERNEL_REDUCE, L.MF_F64, ["x", "y"], ["a"], exprs, vec=1))
    assert part.count("mf_dw_sqrt(") == 1
    assert part.count("mf_dw_pow(") == 2 and part.count("mf_dw_logabs(") == 1 and part.count("mf_dw_log(") == 0
    assert part.count("mf_dw_rcp(") == 1


def test_definitions_compare_up_to_operand_order():
    from morefit_gb300.workloads import _definition
    assert _definition("(-(Fl)+1.0)") == _definition("(1.0+-(Fl))")
    assert _definition("(a*b*c)") == _definition("(c*(b*a))")
    assert _definition("(a+-(b))") != _definition("(b+-(a))")
    assert _definition("pow(a,b)") != _definition("pow(b,a)")
    assert _definition("((a==0.0) ? b : c)") != _definition("((a==0.0) ? c : b)")
    assert _definition("1.0/(a)") != _definition("2.0/(a)")


@pytest.mark.gpu
def test_shared_values_equal_their_own_kernels():
    """pow(x, n), pow(x, m), ln x and 1/x of one base in one kernel equal, bit
    for bit, kernels that hold each alone; 1/x^2, there the square of 1/x, is
    within 3e-14. One event per segment, so that every value is seen: positive
    and negative bases (odd, even and fractional exponents), one and zero. A
    segment with a non-finite value is evaluated again in native FP64, whole."""
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0)
    x = np.array([1.0, 0.5, 2.0, 1e-3, 37.25, 1e3, -1.0, -0.5, -2.0, -37.25, 0.0, np.nextafter(1.0, 2.0)])
    exprs = ["pow(x,n)", "pow(x,m)", "log(x)", "1.0/(x)", "1.0/((x*x))"]
    begin, count = np.arange(x.size, dtype=np.uint64), np.ones(x.size, dtype=np.uint32)

    def values(es, n, m):
        blk = CUDABlock(b, np.float64)
        blk.MakeComputeKernel("shared", 0, ["x"], ["r"] * len(es), ["n", "m"], es, True)
        blk.CopyToInputBuffer(x[None, :])
        return blk.SubmitSegments(begin, count, np.tile([n, m], (x.size, 1)))

    for n, m in ((3.0, 2.0), (4.0, -1.0), (2.5, 1.5), (0.0, 0.5), (-3.25, 7.0)):
        got = values(exprs, n, m)
        with np.errstate(all="ignore"):
            ref = np.stack([np.power(x, n), np.power(x, m), np.log(x), 1.0 / x, 1.0 / (x * x)], axis=1)
        finite = np.isfinite(ref).all(axis=1)
        assert np.array_equal(np.isfinite(got).all(axis=1), finite)
        for j, e in enumerate(exprs[:4]):
            assert np.array_equal(got[finite, j], values([e], n, m)[finite, 0]), (e, n, m)
        assert (np.abs(got[finite, 4] - ref[finite, 4]) <= 3e-14 * ref[finite, 4]).all()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 255, 513, 5003])
def test_sums_of_products_match_fp64(n):
    """Sums and differences of products and values, nested and negated, as an
    output of their own, under a logarithm, plus a parameter-only value, and
    used by two outputs: within 1e-12 of the sum of the terms' magnitudes."""
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0, resident_idle_us=0)
    rng = np.random.default_rng(n)
    x, y = rng.uniform(0.5, 1.5, n), rng.uniform(-1.0, 1.0, n)
    a, c = 0.37, -1.25
    s = "((x*y)+-(((y*y)*a))+x+-((c*y)))"
    exprs = ["((x*y)+-((y*y*x))+(x+-(y)))", f"log((7.0+{s}))", "((x*y)+-((y*x*x))+a)", f"({s}*y)", f"({s}+(x*x*x))",
             "-((-((x*x))+-(y)))", "((x+y)+(x*a)+(y*c)+1.5)"]
    blk = CUDABlock(b, np.float64)
    blk.MakeComputeKernel("sums", 0, ["x", "y"], ["r"] * len(exprs), ["a", "c"], exprs, True)
    blk.CopyToInputBuffer(np.stack([x, y]))
    blk.CopyToParameterBuffer([a, c])
    blk.SubmitKernel()
    S = x * y - y * y * a + x - c * y
    ref = np.stack([x * y - y * y * x + (x - y), np.log(7.0 + S), x * y - y * x * x + a, S * y, S + x * x * x, x * x + y,
                    x + y + x * a + y * c + 1.5])
    got = blk.CopyFromKahanBuffer()
    assert (np.abs(got - ref.sum(axis=1)) <= 1e-12 * np.maximum(np.abs(ref).sum(axis=1), 1.0)).all()
    seg = blk.SubmitSegments([0], [n], [[a, c]])[0]
    assert (np.abs(seg - ref.sum(axis=1)) <= 1e-12 * np.maximum(np.abs(ref).sum(axis=1), 1.0)).all()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 257, 5003])
def test_outputs_scaled_by_parameters_match_fp64(n):
    """Outputs with parameter-only factors, which are applied to the sum: a
    column, a product, a function and a sum times one and two of them, plus a
    parameter-only value, and one whose factor is zero: within 1e-12 of the sum
    of the terms' magnitudes."""
    from morefit_gb300.backend import CUDABackend, CUDABlock
    b = CUDABackend(0, resident_idle_us=0)
    rng = np.random.default_rng(n + 7)
    x, y = rng.uniform(0.5, 1.5, n), rng.uniform(-1.0, 1.0, n)
    a, c, z = 0.37, -1.25, 0.0
    exprs = ["(x*a)", "((x*y)*a)", "(a*(c*(x*y)))", "((x*a)+c)", "(c+((x*y*y)*a))", "(sqrt(x)*c)", "(((x*y)+(y*y))*a)",
             "((x*y)*z)", "(((x*y)+(x*x*y)+y)*(a*c))"]
    blk = CUDABlock(b, np.float64)
    blk.MakeComputeKernel("scaled", 0, ["x", "y"], ["r"] * len(exprs), ["a", "c", "z"], exprs, True)
    blk.CopyToInputBuffer(np.stack([x, y]))
    blk.CopyToParameterBuffer([a, c, z])
    blk.SubmitKernel()
    ref = np.stack([x * a, x * y * a, a * c * x * y, x * a + c, c + x * y * y * a, np.sqrt(x) * c, (x * y + y * y) * a,
                    0.0 * x, (x * y + x * x * y + y) * a * c])
    tol = 1e-12 * np.maximum(np.abs(ref).sum(axis=1), 1.0)
    assert (np.abs(blk.CopyFromKahanBuffer() - ref.sum(axis=1)) <= tol).all()
    assert (np.abs(blk.SubmitSegments([0], [n], [[a, c, z]])[0] - ref.sum(axis=1)) <= tol).all()
    b.close()
