"""Split products over patches whose element matrices all equal their transposes read packed units: every element size
of the patch kernel against the oracle, in one launch and in launches per colour, and the same bits as the whole units
(which one asymmetric element makes the operator use) in every row that this element does not reach."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from helpers import FP64_RTOL, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 10, 11, 12])
@pytest.mark.parametrize("n_elem", [1, 33, 700])
def test_packed_products(gpu, n, n_elem, mode):
    rng = np.random.default_rng(100 * n + n_elem)
    n_dofs = max(n + 2, 2 * n_elem)
    # neighbouring elements share DoFs, as on a mesh
    emap = np.stack([(min(2 * e, n_dofs - n) + rng.permutation(n)) for e in range(n_elem)]).astype(np.uint32)
    k = rng.normal(size=(n_elem, n, n))
    ke = k + k.transpose(0, 2, 1)
    assert np.array_equal(ke, ke.transpose(0, 2, 1))
    u = rng.uniform(-1, 1, n_dofs)
    out = []
    for odd in (False, True):
        k2 = ke.copy()
        if odd and n > 1:
            k2[-1, 0, n - 1] = np.nextafter(k2[-1, 0, n - 1], 9.0)
        maps = Maps()
        maps.set_map(n_elem, emap, n, n_dofs)
        A = aMatFree(maps)
        A.set_precision(PRECISION.FP64_SPLIT)
        A.set_patch_mode(mode)
        A.set_element_matrices(0, k2)
        A.finalize()
        v = np.empty(n_dofs)
        A.matvec(v, u, True)
        assert rel(v, oracle.Problem(n_dofs, emap, k2).matvec(u)) < FP64_RTOL
        out.append(v)
    far = np.ones(n_dofs, dtype=bool)
    far[emap[-1]] = False
    assert np.array_equal(out[0][far], out[1][far])
