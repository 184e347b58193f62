"""Double-float products from the corrected symmetric arena, whose terms run in pairs: each pair of entries alone, and
entries over 14 orders of magnitude within the arena's bound per row, in formats 3 (FP64 u) and 4 (FP32 u)."""
import numpy as np
import pytest
import torch

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree

pytestmark = pytest.mark.gpu


def product(emap, ke, u, fmt):
    maps = Maps()
    maps.set_map(len(emap), emap, emap.shape[1], len(u))
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_symmetric_inner(fmt)
    A.set_element_matrices(0, ke)
    A.finalize()
    du = torch.from_numpy(u).cuda()
    dv = torch.empty_like(du)
    torch.cuda.synchronize()
    A.matvec_inner_device(dv.data_ptr(), du.data_ptr())
    torch.cuda.synchronize()
    return dv.cpu().numpy()


@pytest.mark.parametrize("fmt", [3, 4])
@pytest.mark.parametrize("n", [20, 24, 30, 60, 18, 37])
def test_single_pairs(gpu, n, fmt):
    r, c = np.triu_indices(n)
    n_elem = len(r)
    emap = np.arange(n_elem * n, dtype=np.uint32).reshape(n_elem, n)
    ke = np.zeros((n_elem, n, n))
    e = np.arange(n_elem)
    ke[e, r, c] = ke[e, c, r] = 1.0 + e / 7.0
    u = np.random.default_rng(n).uniform(0.5, 1, n_elem * n).astype(np.float32).astype(float)
    v = product(emap, ke, u, fmt).reshape(n_elem, n)
    ref = np.einsum("eij,ej->ei", ke, u.reshape(n_elem, n))
    assert np.all(v[ref == 0] == 0)
    assert np.all(np.abs(v - ref) <= 2.0 ** -32 * np.abs(ref))  # (an entry: 24 bits and 8 of the rest, 2^-33)


@pytest.mark.parametrize("fmt", [3, 4])
@pytest.mark.parametrize("n_elem", [1, 7, 700])
@pytest.mark.parametrize("n", [20, 24, 30, 60, 37])
def test_rows_within_their_bound(gpu, n, n_elem, fmt):
    rng = np.random.default_rng(n + n_elem)
    n_dofs = n_elem * (n // 2) + n
    emap = np.stack([e * (n // 2) + rng.permutation(n) for e in range(n_elem)]).astype(np.uint32)
    k = rng.normal(size=(n_elem, n, n)) * 10.0 ** rng.uniform(-7, 7, (n_elem, n, n))
    ke = k + k.transpose(0, 2, 1)
    u = (rng.normal(size=n_dofs) * 10.0 ** rng.uniform(-3, 3, n_dofs)).astype(np.float32).astype(float)
    v = product(emap, ke, u, fmt)
    ref = oracle.Problem(n_dofs, emap, ke).matvec(u)
    size = oracle.Problem(n_dofs, emap, np.abs(ke)).matvec(np.abs(u))
    # 2^-33 per entry; the double-float sums add (8 n + 10) 2^-48, far below
    assert np.all(np.abs(v - ref) <= 2.0 ** -32 * size + 2.0 ** -95 * np.abs(ke).max() * np.abs(u).max() * n)
