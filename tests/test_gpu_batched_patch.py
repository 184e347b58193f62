"""The batched product over patches: each kernel (element size, arithmetic, width of the column block) against the
oracle column by column, at column counts that fill a block, part of one and several, padded rows, constrained
columns, DoFs that no element lists, patches of one element, and random maps; repeated calls bit for bit; the launches
per colour that a caller's capture records agree."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from amat_gb300 import problems as P
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu

FP32_RTOL = 1e-5


def products(n_dofs, emap, ke, fixed, nrhs, ld, f32, prec=PRECISION.FP64_SPLIT):
    import torch
    maps = Maps()
    maps.set_map(len(emap), emap, emap.shape[1], n_dofs)
    maps.set_bdr_map(fixed, np.zeros(len(fixed)))
    A = aMatFree(maps)
    A.set_precision(prec)
    A.set_element_matrices(0, ke)
    A.finalize()
    dt = torch.float32 if f32 else torch.float64
    U = torch.tensor(np.random.default_rng(nrhs).uniform(-1, 1, (n_dofs, ld)), dtype=dt, device="cuda")
    pr = oracle.Problem(n_dofs, emap, ke, fixed, np.zeros(len(fixed)))
    tol = FP32_RTOL if f32 else FP64_RTOL
    u = U.double().cpu().numpy()
    for bc in (False, True):
        V, W = torch.full_like(U, 7.0), torch.full_like(U, 7.0)
        A.matvec_batched_device(V.data_ptr(), U.data_ptr(), nrhs, ld, f32=f32, bc=bc)
        A.matvec_batched_device(W.data_ptr(), U.data_ptr(), nrhs, ld, f32=f32, bc=bc)
        A.synchronize()
        assert torch.equal(V[:, :nrhs], W[:, :nrhs])
        v = V.double().cpu().numpy()
        for j in sorted({0, 1, nrhs // 2, nrhs - 1}):
            ref = pr.matmult_bc(u[:, j]) if bc else pr.matvec(u[:, j])
            assert rel(v[:, j], ref) < tol, (bc, j)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.matvec_batched_device(W.data_ptr(), U.data_ptr(), nrhs, ld, f32=f32, bc=True,
                                stream=torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    assert rel(W[:, :nrhs].double().cpu().numpy(), v[:, :nrhs]) < tol


@pytest.mark.parametrize("nrhs,pad", [(4, 0), (8, 4), (16, 0), (20, 0), (32, 4), (36, 0), (64, 0), (100, 0)])
@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("kind,shape", [(P.HEX8_ELASTIC, (5, 4, 7)), (P.TET10_ELASTIC, (3, 2, 3)),
                                        (P.HEX20_ELASTIC, (3, 2, 3))])
def test_patch_products(gpu, kind, shape, f32, nrhs, pad):
    m = P.Mesh(kind, *shape, jitter=0.1, seed=5)
    ke = m.element_matrices(ngt=3 if kind == P.HEX20_ELASTIC else 2)
    fixed = np.arange(0, m.n_dofs, 11, dtype=np.uint64)
    products(m.n_dofs, m.dof_map(), ke, fixed, nrhs, nrhs + pad, f32)


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("n", [24, 30, 60])
def test_patch_products_of_random_maps(gpu, n, f32):
    """Single-DoF lists, DoFs shared by many patches or by none, DoFs in no element."""
    rng = np.random.default_rng(n)
    n_dofs = 340
    emap = np.stack([rng.choice(n_dofs - 5, size=n, replace=False) for _ in range(41)]).astype(np.uint32)
    ke = rng.normal(size=(41, n, n))
    products(n_dofs, emap, ke, np.array([2, 3, 50, n_dofs - 1], dtype=np.uint64), 24, 24, f32)
    products(n_dofs, emap[:1], ke[:1], np.array([2], dtype=np.uint64), 12, 12, f32)


def test_patch_products_of_an_fp32_operator(gpu):
    m = P.Mesh(P.HEX8_ELASTIC, 6, jitter=0.1, seed=5)
    products(m.n_dofs, m.dof_map(), m.element_matrices(), np.zeros(0, np.uint64), 32, 32, True, PRECISION.FP32)
