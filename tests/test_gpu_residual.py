"""Residuals in FP64 between the FP32 segments of a mixed solve, and the update of the recursion there: the reported
residual against numpy, a solve of many short segments, breakdown in the first one; sizes around one block of the
vector passes and their unrolled steps."""
import numpy as np
import pytest

from amat_gb300 import problems as P
from test_gpu_cg_iteration import operator

pytestmark = pytest.mark.gpu

SHAPES = [(P.HEX8_POISSON, (1, 1, 1)), (P.HEX8_POISSON, (5, 5, 6)), (P.TET10_POISSON, (7, 7, 7)),
          (P.HEX8_POISSON, (23, 22, 21)), (P.TET10_POISSON, (4, 3, 3))]


@pytest.mark.parametrize("kind,shape", SHAPES)
def test_reported_residual(gpu, kind, shape):
    A, pr, b = operator(kind, shape)
    b = b + 1.0  # (also on constrained rows)
    for mixed in (False, True):
        if mixed:
            x, st = A.solve_mixed(b, rtol=1e-3, inner_rtol=0.1)
        else:
            x, st = A.solve(b, rtol=1e-3, atol=0.0)
        r = np.linalg.norm(b - pr.matmult_bc(x)) / np.linalg.norm(b)
        # each side's A x is within some 1e-16 |A| |x|, which is below 1e4 |b| here
        assert st.status == 0 and abs(st.rel_residual - r) <= 1e-11


@pytest.mark.parametrize("inner_rtol", [0.3, 0.999, 1.0])
@pytest.mark.parametrize("kind,shape", SHAPES)
def test_segments(gpu, kind, shape, inner_rtol):
    """inner_rtol near 1: segments that end after an iteration or two, each with an update of the recursion."""
    A, pr, b = operator(kind, shape)
    x, st = A.solve_mixed(b, rtol=1e-9, inner_rtol=inner_rtol, max_outer=2000, max_inner=3, raise_on_fail=False)
    if st.status == 0:
        assert np.linalg.norm(b - pr.matmult_bc(x)) <= 1.01e-9 * np.linalg.norm(b)
    else:
        assert inner_rtol == 1.0


def test_breakdown_in_a_segment(gpu):
    A, pr, b = operator(P.HEX8_POISSON, (5, 5, 5), sign=-1.0)
    with pytest.raises(RuntimeError):
        A.solve_mixed(b, rtol=1e-8)
