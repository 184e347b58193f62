"""Matrix-free products over every quadrature rule (1, 2 and 3 points per direction: 8 or 32 lanes an element) and
element kind, from one element to several rounds per warp, with constrained DoFs: against the oracle's product of the
same rule's element matrices; the launches per colour that a caller's capture records give the same bits."""
import numpy as np
import pytest

import oracle
from amat_gb300 import MATFREE_TYPE, Maps, aMatFree
from amat_gb300 import problems as P
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu

FP32_RTOL = 1e-5  # as for the other FP32 matrix-free products


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 5), (26, 24, 22)])
@pytest.mark.parametrize("ngt", [1, 2, 3])
@pytest.mark.parametrize("kind", [P.HEX8_POISSON, P.HEX8_ELASTIC, P.HEX20_ELASTIC, P.TET10_POISSON, P.TET10_ELASTIC])
def test_products_of_every_rule(gpu, kind, ngt, shape):
    import torch
    if shape[0] > 20 and kind not in (P.HEX8_POISSON, P.HEX8_ELASTIC):
        shape = (9, 8, 7)
    m = P.Mesh(kind, *shape, jitter=0.1, seed=5)
    fixed = np.arange(0, m.n_dofs, 7, dtype=np.uint64)
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    maps.set_bdr_map(fixed, np.zeros(len(fixed)))
    A = aMatFree(maps)
    A.set_matfree_type(MATFREE_TYPE.FREE)
    A.set_element_kind(kind, 1.0, 0.3, ngt)
    A.set_element_coords(0, m.coords[m.elem_nodes])
    A.finalize()
    pr = oracle.Problem(m.n_dofs, m.dof_map(), m.element_matrices(ngt=ngt), fixed, np.zeros(len(fixed)))
    u = torch.tensor(np.random.default_rng(ngt).uniform(-1, 1, m.n_dofs), device="cuda")
    for call, x, tol in [(A.matmult_bc_device, u, FP64_RTOL), (A.matmult_bc_device_f32, u.float(), FP32_RTOL)]:
        v, w = torch.full_like(x, 7.0), torch.full_like(x, 8.0)
        call(v.data_ptr(), x.data_ptr())
        A.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(w.data_ptr(), x.data_ptr(), torch.cuda.current_stream().cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(v, w)
        assert rel(v.double().cpu().numpy(), pr.matmult_bc(x.double().cpu().numpy())) < tol
