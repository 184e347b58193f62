"""What the operator says of a product: the kernels that it launches, and the bytes of its matrices in the form that it
reads."""
import pytest

from amat_gb300 import MATFREE_TYPE, PRECISION, Maps, aMatFree
from amat_gb300 import problems as P

pytestmark = pytest.mark.gpu


def operator(m, how, ngt):
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    A = aMatFree(maps)
    if how == "free":
        A.set_matfree_type(MATFREE_TYPE.FREE)
        A.set_element_kind(m.kind, 1.0, 0.3, ngt)
        A.set_element_coords(0, m.coords[m.elem_nodes])
    else:
        A.set_precision(how)
        A.set_element_matrices(0, m.element_matrices(ngt=ngt))
    A.finalize()
    return A


@pytest.mark.parametrize("kind,n,jitter,how,kernels,per", [
    (P.HEX20_ELASTIC, 12, 0.1, PRECISION.FP64_SPLIT, 3, 22080),  # block units: max|u|, elements, gather pass
    (P.HEX20_ELASTIC, 12, 0.0, PRECISION.FP64_SPLIT, 3, 28800),  # a regular mesh: pairs of rounding, whole matrices
    (P.HEX20_ELASTIC, 4, 0.1, PRECISION.FP64_SPLIT, 3, 28800),   # few elements: whole matrices
    (P.HEX20_ELASTIC, 4, 0.1, PRECISION.FP64, 2, 28800),         # elements, gather pass
    (P.HEX8_ELASTIC, 8, 0.1, PRECISION.FP64_SPLIT, 3, 4608),
    (P.HEX8_ELASTIC, 8, 0.1, PRECISION.FP32, 2, 2304),
    (P.HEX8_ELASTIC, 8, 0.1, "free", 2, 192),
    (P.TET10_POISSON, 8, 0.1, PRECISION.FP64_SPLIT, 2, None),    # patches, combine pass
    (P.TET10_POISSON, 8, 0.1, PRECISION.FP64, 2, None),
])
def test_cost(gpu, kind, n, jitter, how, kernels, per):
    m = P.Mesh(kind, n, jitter=jitter, seed=3)
    A = operator(m, how, 3 if kind == P.HEX20_ELASTIC else 2)
    got, moved = A.product_cost()
    assert got == kernels
    vec = 2 * m.n_dofs * (4 if how == PRECISION.FP32 else 8)
    info = A.info()
    if per:
        assert moved == m.n_elem * (per + 4 * m.ndpe) + vec
    else:
        assert vec < moved <= info["ke_bytes"] + info["patch_index_bytes"] + vec
        # symmetric bit for bit: packed triangles in the split arithmetic
        assert (moved < info["ke_bytes"]) == (how == PRECISION.FP64_SPLIT)


def test_before_finalize(gpu):
    from amat_gb300._native import AfmError
    m = P.Mesh(P.HEX8_ELASTIC, 2)
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    A = aMatFree(maps)
    with pytest.raises(AfmError):
        A.product_cost()
