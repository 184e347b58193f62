"""Split products over patches scale u by a power of two per patch: u whose size changes by hundreds of orders of
magnitude across the mesh keeps its accuracy everywhere, zero and subnormal regions stay exact, and a product in one
launch writes the constrained rows and the DoFs that no element lists."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from amat_gb300 import problems as P

pytestmark = pytest.mark.gpu


def operator(m, ke, extra, fixed, mode):
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs + extra)
    maps.set_bdr_map(fixed, np.zeros(len(fixed)))
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_patch_mode(mode)
    A.set_element_matrices(0, ke)
    A.finalize()
    return A


@pytest.mark.parametrize("mode", [2, 3])
@pytest.mark.parametrize("kind,shape,span", [(P.HEX8_POISSON, (40, 6, 5), 0.3), (P.TET10_POISSON, (14, 4, 3), 0.5)])
def test_u_over_many_orders_of_magnitude(gpu, kind, shape, span, mode):
    m = P.Mesh(kind, *shape, jitter=0.1, seed=3)
    ke = m.element_matrices()
    A = operator(m, ke, 0, np.zeros(0, np.uint64), mode)
    x = m.coords[:, 0]
    u = np.random.default_rng(2).uniform(0.5, 1, m.n_dofs) * 2.0 ** np.round(-200 * np.abs(x - 0.4))
    u[x > 0.9] = 0.0
    v = np.empty(m.n_dofs)
    A.matvec(v, u, True)
    pr = oracle.Problem(m.n_dofs, m.dof_map(), ke)
    ref, size = pr.matvec(u), oracle.Problem(m.n_dofs, m.dof_map(), np.abs(ke)).matvec(np.abs(u))
    # row by row: the split arithmetic's bound (8 n + 10) 2^-48 |K||u| with n = 10, and the 2^-98 of its patch's
    # largest |u| that an entry may lose (a patch spans less than `span` along x)
    lost = np.array([np.abs(u[np.abs(x - t) <= span]).max() for t in np.unique(x)])[np.unique(x, return_inverse=True)[1]]
    assert np.all(np.abs(v - ref) <= 90 * 2.0 ** -48 * size + 64 * np.abs(ke).max() * 2.0 ** -98 * lost)
    far = x > 0.98
    assert np.all(v[far] == 0.0)


@pytest.mark.parametrize("mode", [2, 3])
def test_unlisted_and_constrained_dofs(gpu, mode):
    m = P.Mesh(P.HEX8_POISSON, 7, 6, 5, jitter=0.1, seed=3)
    ke = m.element_matrices()
    for extra in (0, 5):
        n = m.n_dofs + extra
        fixed = np.array([0, 3, 100, n - 1], dtype=np.uint64)
        A = operator(m, ke, extra, fixed, mode)
        u = np.random.default_rng(4).uniform(-1, 1, n)
        v = np.full(n, np.nan)
        A.matmult_bc(v, u)
        ref = oracle.Problem(n, m.dof_map(), ke, fixed, np.zeros(4)).matmult_bc(u)
        assert np.linalg.norm(v - ref) < 1e-12 * np.linalg.norm(ref)
        assert np.array_equal(v[fixed.astype(int)], u[fixed.astype(int)])
        A.matvec(v, u, True)
        assert np.all(v[m.n_dofs:] == 0.0)
