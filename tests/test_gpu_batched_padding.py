"""Columns of a batched product beyond nrhs are zero after every call, whichever way it runs."""
import numpy as np
import pytest

from amat_gb300 import Maps, aMatFree
from amat_gb300 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nrhs,ld", [(4, 8), (16, 20), (32, 64)])
def test_padding_columns(gpu, nrhs, ld, f32):
    import torch
    m = P.Mesh(P.HEX8_ELASTIC, 10, jitter=0.1, seed=2)
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    A = aMatFree(maps)
    A.set_element_matrices(0, m.element_matrices())
    A.finalize()
    U = torch.tensor(np.random.default_rng(1).uniform(-1, 1, (m.n_dofs, ld)), device="cuda",
                     dtype=torch.float32 if f32 else torch.float64)
    for patches in (1, 0, 2):
        A.set_batch_patches(patches)
        for _ in range(2):
            V = torch.full_like(U, 7.0)
            torch.cuda.synchronize()
            A.matvec_batched_device(V.data_ptr(), U.data_ptr(), nrhs, ld, f32=f32)
            A.synchronize()
            assert torch.all(V[:, nrhs:] == 0.0)
            assert torch.any(V[:, :nrhs] != 0.0)
