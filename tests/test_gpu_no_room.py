"""Buffers that only make products faster may find no room on the device: the operator does without them, with the same
results, whichever of them fails."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from amat_gb300 import problems as P
from amat_gb300._native import check
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu


def operator(m, ke):
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_element_matrices(0, ke)
    return A


def fail(A, skip, count):
    check(A._lib.afm_debug_fail_allocations(A._h, skip, count), "afm_debug_fail_allocations")


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("skip,count", [(0, 1), (1, 1), (2, 1), (3, 1), (4, 1), (0, 5)])
def test_batched_plan(gpu, skip, count, f32):
    import torch
    m = P.Mesh(P.HEX8_ELASTIC, 6, 5, 7, jitter=0.1, seed=2)
    ke = m.element_matrices()
    A = operator(m, ke)
    A.finalize()
    U = torch.tensor(np.random.default_rng(skip).uniform(-1, 1, (m.n_dofs, 16)), device="cuda",
                     dtype=torch.float32 if f32 else torch.float64)
    pr = oracle.Problem(m.n_dofs, m.dof_map(), ke)
    u = U.double().cpu().numpy()
    fail(A, skip, count)
    for nrhs in (8, 16, 16):
        V = torch.full_like(U, float("nan"))
        A.matvec_batched_device(V.data_ptr(), U.data_ptr(), nrhs, 16, f32=f32)
        A.synchronize()
        v = V.double().cpu().numpy()
        for j in (0, nrhs - 1):
            assert rel(v[:, j], pr.matvec(u[:, j])) < (1e-5 if f32 else FP64_RTOL)
    fail(A, 0, 0)
