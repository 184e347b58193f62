"""The patch kernels of the batched products, taken whatever the autotuner would choose: each element size and arithmetic
against the oracle column by column, the same bits again and in a solve's captured graph; the modes of the choice."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from amat_gb300 import problems as P
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu


def operator(m, ke, fixed):
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    maps.set_bdr_map(fixed, np.zeros(len(fixed)))
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_element_matrices(0, ke)
    A.finalize()
    return A


@pytest.mark.parametrize("kind,shape,f32,has", [
    (P.HEX8_ELASTIC, (5, 4, 7), False, True), (P.HEX8_ELASTIC, (5, 4, 7), True, True),
    (P.TET10_ELASTIC, (3, 2, 3), False, True), (P.TET10_ELASTIC, (3, 2, 3), True, True),
    (P.HEX20_ELASTIC, (3, 2, 3), True, True), (P.HEX20_ELASTIC, (3, 2, 3), False, False)])
@pytest.mark.parametrize("nrhs,ld", [(4, 4), (16, 20), (20, 20), (36, 36), (64, 64)])
def test_forced(gpu, kind, shape, f32, has, nrhs, ld):
    import torch
    m = P.Mesh(kind, *shape, jitter=0.1, seed=7)
    ke = m.element_matrices(ngt=3 if kind == P.HEX20_ELASTIC else 2)
    fixed = np.arange(0, m.n_dofs, 9, dtype=np.uint64)
    A = operator(m, ke, fixed)
    pr = oracle.Problem(m.n_dofs, m.dof_map(), ke, fixed, np.zeros(len(fixed)))
    U = torch.tensor(np.random.default_rng(nrhs).uniform(-1, 1, (m.n_dofs, ld)), device="cuda",
                     dtype=torch.float32 if f32 else torch.float64)
    u = U.double().cpu().numpy()
    for mode in (2, 0):
        A.set_batch_patches(mode)
        V, W = torch.full_like(U, 7.0), torch.full_like(U, 7.0)
        for out in (V, W):
            A.matvec_batched_device(out.data_ptr(), U.data_ptr(), nrhs, ld, f32=f32, bc=True)
        A.synchronize()
        assert A.batch_patches(nrhs, ld, f32) == (has and mode == 2)
        assert torch.equal(V[:, :nrhs], W[:, :nrhs])
        v = V.double().cpu().numpy()
        for j in sorted({0, 1, nrhs // 2, nrhs - 1}):
            assert rel(v[:, j], pr.matmult_bc(u[:, j])) < (1e-5 if f32 else FP64_RTOL)


@pytest.mark.parametrize("mixed", [False, True])
def test_solve(gpu, mixed):
    import torch
    m = P.Mesh(P.HEX8_ELASTIC, 6, jitter=0.1, seed=7)
    ke = m.element_matrices()
    fixed = np.flatnonzero(np.repeat(m.coords[:, 0] == m.coords[:, 0].min(), 3)).astype(np.uint64)
    A = operator(m, ke, fixed)
    pr = oracle.Problem(m.n_dofs, m.dof_map(), ke, fixed, np.zeros(len(fixed)))
    B = np.random.default_rng(3).standard_normal((m.n_dofs, 8))
    B[fixed.astype(np.int64)] = 0.0
    d_b = torch.tensor(B, device="cuda")
    A.set_batch_patches(2)
    out = []
    for _ in range(2):
        X = torch.zeros_like(d_b)
        torch.cuda.synchronize()
        A.solve_batched_device(d_b.data_ptr(), X.data_ptr(), 8, rtol=1e-10, mixed=mixed)
        out.append(X)
    assert A.batch_patches(8, solve=mixed)
    assert torch.equal(out[0], out[1])
    x = out[0].cpu().numpy()
    for j in range(8):
        assert rel(pr.matmult_bc(x[:, j]), B[:, j]) < 1e-9


def test_modes(gpu):
    from amat_gb300._native import AfmError
    m = P.Mesh(P.HEX8_ELASTIC, 2, jitter=0.1, seed=7)
    A = operator(m, m.element_matrices(), np.zeros(0, np.uint64))
    for mode in (-1, 3):
        with pytest.raises(AfmError):
            A.set_batch_patches(mode)
    with pytest.raises(AfmError):
        A.batch_patches(8)
