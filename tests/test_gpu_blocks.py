"""Split products on block units (elements of 60 DoFs, symmetric up to rounding, from ten per SM up): each pair of entries
alone, entries over 14 orders of magnitude within the split arithmetic's bound per row, differences between K and its
transpose that the units hold and those for which the operator keeps whole matrices, colours in one launch and in
launches of their own."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from amat_gb300 import problems as P
from helpers import rel
from test_gpu_pairs import product

pytestmark = pytest.mark.gpu


def test_single_pairs(gpu):
    """Element e holds one pair of entries (or one diagonal entry); every pair of the matrix has its element."""
    n = 60
    r, c = np.triu_indices(n)
    n_elem = len(r)
    emap = np.arange(n_elem * n, dtype=np.uint32).reshape(n_elem, n)
    ke = np.zeros((n_elem, n, n))
    e = np.arange(n_elem)
    ke[e, r, c] = ke[e, c, r] = 1.0 + e / 7.0
    u = np.random.default_rng(n).uniform(0.5, 1, n_elem * n)
    v = product(emap, ke, u).reshape(n_elem, n)
    ref = np.einsum("eij,ej->ei", ke, u.reshape(n_elem, n))
    assert np.all(v[ref == 0] == 0)
    assert np.all(np.abs(v - ref) <= 2.0 ** -45 * np.abs(ref))


@pytest.mark.parametrize("n_elem", [1519, 1520, 1823, 1825, 3001])
def test_rows_within_their_bound(gpu, n_elem):
    n = 60
    rng = np.random.default_rng(n_elem)
    n_dofs = n_elem * (n // 2) + n
    emap = np.stack([e * (n // 2) + rng.permutation(n) for e in range(n_elem)]).astype(np.uint32)
    k = rng.normal(size=(n_elem, n, n)) * 10.0 ** rng.uniform(-7, 7, (n_elem, n, n))
    ke = k + k.transpose(0, 2, 1)
    u = rng.normal(size=n_dofs) * 10.0 ** rng.uniform(-3, 3, n_dofs)
    v = product(emap, ke, u)
    ref = oracle.Problem(n_dofs, emap, ke).matvec(u)
    size = oracle.Problem(n_dofs, emap, np.abs(ke)).matvec(np.abs(u))
    # (8 n + 10) 2^-48 per element row, the FP64 sums of two elements, and 2^-98 of max|u| per entry
    assert np.all(np.abs(v - ref) <= (8 * n + 14) * 2.0 ** -48 * size + 2.0 ** -95 * np.abs(ke).max() * np.abs(u).max() * n)


@pytest.mark.parametrize("ulps", [1, 16, 2.0 ** 7, 2.0 ** 8, 2.0 ** 20])
def test_nearly_symmetric(gpu, ulps):
    """K(r, c) and K(c, r) differ by up to `ulps` 2^-53 of the diagonal entries (held up to 2^-46, else whole matrices):
    the antisymmetric part alone, found as the difference of two products, is the oracle's."""
    n, n_elem = 60, 1600
    rng = np.random.default_rng(int(ulps))
    n_dofs = n_elem * n
    emap = np.arange(n_dofs, dtype=np.uint32).reshape(n_elem, n)
    # few significant bits, so that the products and leading sums of the split arithmetic are exact
    s = rng.integers(-8, 9, (n_elem, n, n)).astype(float)
    s = s + s.transpose(0, 2, 1)
    s[:, np.arange(n), np.arange(n)] = 32.0
    a = np.tril(rng.integers(-1, 2, (n_elem, n, n)), -1) * (ulps * 32.0 * 2.0 ** -53)
    # a where s is 0: elsewhere the split pair (2^-48 of the entry) would not hold the smallest
    ke = s + np.where(s == 0, a, 0.0)
    u = rng.integers(-4, 5, n_dofs).astype(float)
    diff = product(emap, ke, u) - product(emap, s, u)
    ref = np.einsum("eij,ej->ei", ke - s, u.reshape(n_elem, n)).ravel()
    # FP64 rounds the sums, of up to 4 n 16, to 2^-53 of them; the entry's byte to 2^-53 of 32, times 4 and n terms; the
    # low parts' sums add n roundings of 2^-24 of their size
    assert np.all(np.abs(diff - ref) <= n * 64 * 2.0 ** -53 + n * 128 * 2.0 ** -53 + n * 2.0 ** -24 * np.abs(a).max() * 4 * n)


@pytest.mark.parametrize("bc", [False, True])
def test_colours(gpu, bc):
    """One launch for all elements, and all colours in one cooperative launch: the same bits, the oracle's product."""
    m = P.Mesh(P.HEX20_ELASTIC, 12, jitter=0.1, seed=6)
    ke = m.element_matrices(ngt=3)
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    dofs = np.arange(0, m.n_dofs, 17, dtype=np.uint64) if bc else np.zeros(0, np.uint64)
    maps.set_bdr_map(dofs, np.ones(len(dofs)))
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_element_matrices(0, ke)
    A.finalize()
    u = np.random.default_rng(3).uniform(-1, 1, m.n_dofs)
    pr = oracle.Problem(m.n_dofs, m.dof_map(), ke, dofs, np.ones(len(dofs)))
    out = []
    for fused in (0, 1):
        A.set_fused_colours(fused)
        v = np.empty(m.n_dofs)
        if bc:
            A.matmult_bc(v, u)
        else:
            A.matvec(v, u, True)
        assert rel(v, pr.matmult_bc(u) if bc else pr.matvec(u)) < 1e-13
        out.append(v)
    assert np.array_equal(out[0], out[1])
