"""Plans of one element size run every element in one launch and sum the element products per DoF in a second pass:
the same bits as one launch per colour (which a caller's stream capture still records), whole-node and single-DoF
lists, constrained rows written by the pass, DoFs that no element lists, and products on several streams in turn."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from amat_gb300 import problems as P
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu


def mesh_operator(kind, n, prec):
    m = P.Mesh(kind, n, jitter=0.1, seed=6)
    ke = m.element_matrices(ngt=3 if kind == P.HEX20_ELASTIC else 2)
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    dofs, vals = m.boundary_conditions()
    maps.set_bdr_map(dofs, vals)
    A = aMatFree(maps)
    A.set_precision(prec)
    A.set_element_matrices(0, ke)
    A.finalize()
    return m, ke, dofs, vals, A


def captured(call):
    """The call recorded on a caller's stream and replayed once."""
    import torch
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()


@pytest.mark.parametrize("prec", [PRECISION.FP64, PRECISION.FP64_SPLIT])
@pytest.mark.parametrize("kind,n", [(P.HEX20_ELASTIC, 2), (P.HEX20_ELASTIC, 8), (P.HEX8_ELASTIC, 10),
                                    (P.TET10_ELASTIC, 4)])
def test_gather_equals_colour_launches(gpu, kind, n, prec):
    import torch
    m, ke, dofs, vals, A = mesh_operator(kind, n, prec)
    assert A.info()["n_launches"] == 3
    pr = oracle.Problem(m.n_dofs, m.dof_map(), ke, dofs, vals)
    u = torch.tensor(np.random.default_rng(n).uniform(-1, 1, m.n_dofs), device="cuda")
    u32 = u.float()
    calls = [(A.matvec_device, u, pr.matvec(u.cpu().numpy()), FP64_RTOL),
             (A.matmult_bc_device, u, pr.matmult_bc(u.cpu().numpy()), FP64_RTOL)]
    if prec == PRECISION.FP64_SPLIT:
        ref32 = pr.matmult_bc(u32.double().cpu().numpy())
        calls += [(A.matmult_bc_device_f32, u32, ref32, 1e-5)]
    for fmt in (1, 2) if prec == PRECISION.FP64_SPLIT else (1,):
        A.set_symmetric_inner(fmt)
        for call, x, ref, tol in calls:
            v, w = torch.full_like(x, 7.0), torch.full_like(x, 8.0)
            call(v.data_ptr(), x.data_ptr())
            A.synchronize()
            captured(lambda s: call(w.data_ptr(), x.data_ptr(), s))
            assert torch.equal(v, w)
            assert rel(v.cpu().double().numpy(), ref) < tol
    if prec == PRECISION.FP64_SPLIT:
        for fmt in (3, 4, 5):
            A.set_symmetric_inner(fmt)
            v, w = torch.full_like(u, 7.0), torch.full_like(u, 8.0)
            A.matvec_inner_device(v.data_ptr(), u.data_ptr())
            A.synchronize()
            captured(lambda s: A.matvec_inner_device(w.data_ptr(), u.data_ptr(), s))
            assert torch.equal(v, w)


@pytest.mark.parametrize("prec", [PRECISION.FP64, PRECISION.FP64_SPLIT, PRECISION.FP32])
@pytest.mark.parametrize("n", [17, 18, 24, 33, 96])
def test_gather_of_scattered_dofs(gpu, n, prec):
    """Random maps of one element size (one list per DoF, up to dozens of entries), some DoFs in no element."""
    import torch
    rng = np.random.default_rng(n)
    n_dofs, n_elem = 403, 70
    emap = np.stack([rng.choice(n_dofs - 3, size=n, replace=False) for _ in range(n_elem)]).astype(np.uint32)
    ke = rng.normal(size=(n_elem, n, n))
    fixed = np.array([0, 5, n_dofs - 1], dtype=np.uint64)
    maps = Maps()
    maps.set_map(n_elem, emap, n, n_dofs)
    maps.set_bdr_map(fixed, np.zeros(3))
    A = aMatFree(maps)
    A.set_precision(prec)
    A.set_element_matrices(0, ke)
    A.finalize()
    f32 = prec == PRECISION.FP32
    u = torch.tensor(rng.uniform(-1, 1, n_dofs), device="cuda", dtype=torch.float32 if f32 else torch.float64)
    v = torch.full_like(u, float("nan"))
    (A.matmult_bc_device_f32 if f32 else A.matmult_bc_device)(v.data_ptr(), u.data_ptr())
    A.synchronize()
    ref = oracle.Problem(n_dofs, emap, ke, fixed, np.zeros(3)).matmult_bc(u.double().cpu().numpy())
    assert rel(v.double().cpu().numpy(), ref) < (1e-5 if f32 else FP64_RTOL)


def test_products_on_streams_in_turn(gpu):
    """Products of one operator on the operator's and two callers' streams, none waiting on the host, share the
    element-product buffer without mixing their results."""
    import torch
    m, ke, dofs, vals, A = mesh_operator(P.HEX8_ELASTIC, 24, PRECISION.FP64)
    us = [torch.tensor(np.random.default_rng(k).uniform(-1, 1, m.n_dofs), device="cuda") for k in range(3)]
    refs = []
    for x in us:
        v = torch.empty_like(x)
        A.matvec_device(v.data_ptr(), x.data_ptr())
        A.synchronize()
        refs.append(v)
    streams = [None, torch.cuda.Stream(), torch.cuda.Stream()]
    outs = [[torch.empty_like(x) for x in us] for _ in range(20)]
    torch.cuda.synchronize()
    for o in outs:
        for k, s in enumerate(streams):
            A.matvec_device(o[k].data_ptr(), us[k].data_ptr(), s.cuda_stream if s else None)
    torch.cuda.synchronize()
    for o in outs:
        for k in range(3):
            assert torch.equal(o[k], refs[k])
