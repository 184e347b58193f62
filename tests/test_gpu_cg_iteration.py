"""The two launches of a CG iteration and the dot product in the pass before them: iterates against a plain numpy
Jacobi-PCG after every count of iterations around the captured batch (8, an even and an odd number), one block and
many, products with and without the fused dot product (more than 2^18 DoFs), breakdown, and FP64-checked solves."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from amat_gb300 import problems as P
from helpers import rel

pytestmark = pytest.mark.gpu


def operator(kind, shape, sign=1.0, prec=PRECISION.AUTO):
    m = P.Mesh(kind, *shape, jitter=0.1, seed=8)
    ke = sign * m.element_matrices(ngt=3 if kind == P.HEX20_ELASTIC else 2)
    dofs, vals = m.boundary_conditions()
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    maps.set_bdr_map(dofs, vals)
    A = aMatFree(maps)
    A.set_precision(prec)
    A.set_element_matrices(0, ke)
    A.finalize()
    b = np.random.default_rng(1).normal(size=m.n_dofs)
    b[dofs.astype(int)] = 0.0
    return A, oracle.Problem(m.n_dofs, m.dof_map(), ke, dofs, vals), b


@pytest.mark.parametrize("prec", [PRECISION.FP64, PRECISION.FP64_SPLIT])
@pytest.mark.parametrize("kind,shape", [(P.HEX8_POISSON, (3, 3, 3)), (P.HEX8_POISSON, (17, 16, 19)),
                                        (P.HEX8_ELASTIC, (6, 6, 6)), (P.TET10_POISSON, (9, 8, 7))])
def test_iterates(gpu, kind, shape, prec):
    A, pr, b = operator(kind, shape, prec=prec)
    d = A.get_diagonal()
    x, r = np.zeros_like(b), b.copy()
    z = r / d
    p, rz = z.copy(), r @ z
    for k in range(1, 18):
        q = pr.matmult_bc(p)
        a = rz / (p @ q)
        x, r = x + a * p, r - a * q
        z = r / d
        rz, old = r @ z, rz
        p = z + rz / old * p
        if np.linalg.norm(r) <= 1e-6 * np.linalg.norm(b):
            break  # (rounding grows from here on)
        if k in (1, 2, 7, 8, 9, 16, 17):
            y, st = A.solve(b, rtol=1e-14, atol=0.0, maxit=k, raise_on_fail=False)
            assert st.iterations == k
            # each iteration multiplies rounding (1e-15 of the iterate) by a few units at most
            assert rel(y, x) < 1e-15 * 8.0 ** min(k, 5)


@pytest.mark.parametrize("kind,shape", [(P.HEX8_POISSON, (64, 64, 64)), (P.HEX8_POISSON, (63, 63, 63)),
                                        (P.HEX8_ELASTIC, (44, 44, 44))])
def test_solves_around_the_fused_dot_limit(gpu, kind, shape):
    A, pr, b = operator(kind, shape)
    x, st = A.solve(b, rtol=1e-7, atol=0.0, maxit=20000)
    assert st.status == 0
    assert np.linalg.norm(b - pr.matmult_bc(x)) <= 1.01e-7 * np.linalg.norm(b)
    y, sm = A.solve_mixed(b, rtol=1e-7, inner_rtol=0.3)
    assert sm.status == 0
    assert np.linalg.norm(b - pr.matmult_bc(y)) <= 1.01e-7 * np.linalg.norm(b)


def test_breakdown_is_reported(gpu):
    """A negative definite operator: p.q < 0 in the first iteration, x unchanged."""
    A, pr, b = operator(P.HEX8_POISSON, (5, 5, 5), sign=-1.0)
    x, st = A.solve(b, rtol=1e-8, atol=0.0, maxit=50, raise_on_fail=False)
    assert st.status == 103 and np.all(x == 0.0)
