"""Batched products on 8-byte entries at the widest blocks that the shared memory of a CTA takes for an element size: three
ring slots and one warp's columns of U fit in 226 KB."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [PRECISION.FP64, PRECISION.FP64_SPLIT])
@pytest.mark.parametrize("n,nrhs", [(60, 4), (60, 24), (60, 56), (60, 116), (60, 120), (60, 128), (60, 144), (48, 188),
                                    (48, 220), (64, 100), (64, 120), (81, 32), (81, 48), (24, 256), (30, 256)])
def test_wide_blocks(gpu, n, nrhs, prec):
    import torch
    rng = np.random.default_rng(n + nrhs)
    n_dofs, n_elem = 400, 23
    emap = np.stack([rng.choice(n_dofs, size=n, replace=False) for _ in range(n_elem)]).astype(np.uint32)
    ke = rng.normal(size=(n_elem, n, n))
    fixed = np.array([1, 7, 350], dtype=np.uint64)
    maps = Maps()
    maps.set_map(n_elem, emap, n, n_dofs)
    maps.set_bdr_map(fixed, np.zeros(3))
    A = aMatFree(maps)
    A.set_precision(prec)
    A.set_element_matrices(0, ke)
    A.finalize()
    U = torch.tensor(rng.uniform(-1, 1, (n_dofs, nrhs)), device="cuda")
    V = torch.full_like(U, 7.0)
    A.matvec_batched_device(V.data_ptr(), U.data_ptr(), nrhs, bc=True)
    A.synchronize()
    pr = oracle.Problem(n_dofs, emap, ke, fixed, np.zeros(3))
    u, v = U.cpu().numpy(), V.cpu().numpy()
    for j in sorted({0, nrhs // 2, nrhs - 1}):
        assert rel(v[:, j], pr.matmult_bc(u[:, j])) < FP64_RTOL
