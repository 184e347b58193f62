"""The split products with rows in pairs (elements of 24, 30 and 60 DoFs): columns and rows that an element reaches
only through one entry, against the oracle entry by entry; entries over 14 orders of magnitude within the split
arithmetic's bound per row; one element, several per ring slot and partial slots."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree

pytestmark = pytest.mark.gpu


def product(emap, ke, u):
    n_dofs = len(u)
    maps = Maps()
    maps.set_map(len(emap), emap, emap.shape[1], n_dofs)
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_element_matrices(0, ke)
    A.finalize()
    v = np.empty(n_dofs)
    A.matvec(v, u, True)
    return v


@pytest.mark.parametrize("n", [24, 30, 60])
def test_single_entries(gpu, n):
    """Element e holds one entry, at row e mod n and column 7 e mod n, so every lane and column group is read alone."""
    n_elem = 2 * n
    emap = np.arange(n_elem * n, dtype=np.uint32).reshape(n_elem, n)
    ke = np.zeros((n_elem, n, n))
    e = np.arange(n_elem)
    ke[e, e % n, 7 * e % n] = 1.0 + e
    u = np.random.default_rng(n).uniform(0.5, 1, n_elem * n)
    v = product(emap, ke, u).reshape(n_elem, n)
    ref = np.zeros_like(v)
    ref[e, e % n] = (1.0 + e) * u.reshape(n_elem, n)[e, 7 * e % n]
    assert np.all(v[ref == 0] == 0)
    assert np.all(np.abs(v - ref) <= 2.0 ** -45 * np.abs(ref))


@pytest.mark.parametrize("n_elem", [1, 2, 3, 607, 1900])
@pytest.mark.parametrize("n", [24, 30, 60])
def test_rows_within_their_bound(gpu, n, n_elem):
    rng = np.random.default_rng(n + n_elem)
    n_dofs = n_elem * (n // 2) + n
    emap = np.stack([e * (n // 2) + rng.permutation(n) for e in range(n_elem)]).astype(np.uint32)
    ke = rng.normal(size=(n_elem, n, n)) * 10.0 ** rng.uniform(-7, 7, (n_elem, n, n))
    u = rng.normal(size=n_dofs) * 10.0 ** rng.uniform(-3, 3, n_dofs)
    v = product(emap, ke, u)
    ref = oracle.Problem(n_dofs, emap, ke).matvec(u)
    size = oracle.Problem(n_dofs, emap, np.abs(ke)).matvec(np.abs(u))
    # (8 n + 10) 2^-48 per element row, the FP64 sums of two elements, and 2^-98 of max|u| per entry
    assert np.all(np.abs(v - ref) <= (8 * n + 14) * 2.0 ** -48 * size + 2.0 ** -95 * np.abs(ke).max() * np.abs(u).max() * n)
