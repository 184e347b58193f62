"""Finalize leaves nothing pending: the operator's stream is idle when it returns, so that a first product on a caller's
own stream finds the gather lists, the buffers and the packed units in place."""
import numpy as np
import pytest

import oracle
from amat_gb300 import MATFREE_TYPE, PRECISION, Maps, aMatFree
from amat_gb300 import problems as P
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,how", [(P.HEX8_ELASTIC, 24, "free"), (P.HEX8_ELASTIC, 24, PRECISION.FP64),
                                        (P.HEX8_ELASTIC, 24, PRECISION.FP64_SPLIT),
                                        (P.HEX20_ELASTIC, 12, PRECISION.FP64_SPLIT),
                                        (P.HEX8_ELASTIC, 24, PRECISION.FP32), (P.TET10_POISSON, 8, PRECISION.FP64_SPLIT)])
def test_first_product_on_a_callers_stream(gpu, kind, n, how):
    import torch
    m = P.Mesh(kind, n, jitter=0.1, seed=4)
    ngt = 3 if kind == P.HEX20_ELASTIC else 2
    ke = m.element_matrices(ngt=ngt)
    f32 = how == PRECISION.FP32
    u = torch.tensor(np.random.default_rng(n).uniform(-1, 1, m.n_dofs), device="cuda",
                     dtype=torch.float32 if f32 else torch.float64)
    v = torch.full_like(u, float("nan"))
    caller = torch.cuda.Stream()
    torch.cuda.synchronize()
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    A = aMatFree(maps)
    if how == "free":
        A.set_matfree_type(MATFREE_TYPE.FREE)
        A.set_element_kind(kind, 1.0, 0.3, ngt)
        A.set_element_coords(0, m.coords[m.elem_nodes])
    else:
        A.set_precision(how)
        A.set_element_matrices(0, ke)
    A.finalize()
    idle = torch.cuda.ExternalStream(A.stream()).query()
    (A.matvec_device_f32 if f32 else A.matvec_device)(v.data_ptr(), u.data_ptr(), caller.cuda_stream)
    caller.synchronize()
    assert idle
    ref = oracle.Problem(m.n_dofs, m.dof_map(), ke).matvec(u.double().cpu().numpy())
    assert rel(v.double().cpu().numpy(), ref) < (1e-5 if f32 else FP64_RTOL)
