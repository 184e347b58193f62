"""A batched product on a caller's stream is enqueued without waiting for the operator's stream, once its plan and its
combine buffer are there."""
import numpy as np
import pytest

from amat_gb300 import Maps, aMatFree
from amat_gb300 import problems as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
def test_enqueued_without_waiting(gpu, f32):
    import torch
    m = P.Mesh(P.HEX8_ELASTIC, 14, jitter=0.1, seed=2)
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    A = aMatFree(maps)
    A.set_element_matrices(0, m.element_matrices())
    A.finalize()
    U = torch.tensor(np.random.default_rng(1).uniform(-1, 1, (m.n_dofs, 32)), device="cuda",
                     dtype=torch.float32 if f32 else torch.float64)
    V, W = torch.empty_like(U), torch.empty_like(U)
    caller, own = torch.cuda.Stream(), torch.cuda.ExternalStream(A.stream())
    torch.cuda.synchronize()
    A.matvec_batched_device(V.data_ptr(), U.data_ptr(), 32, f32=f32, stream=caller.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(own):
        torch.cuda._sleep(400_000_000)
    A.matvec_batched_device(W.data_ptr(), U.data_ptr(), 32, f32=f32, stream=caller.cuda_stream)
    busy = not own.query()
    torch.cuda.synchronize()
    assert busy
    assert torch.equal(V, W)
