"""Split products on block units hold every entry as the split pair does: with u one entry per element, each row is that
entry's product to 2^-44 of it, in both triangles, for small entries of matrices that are symmetric up to rounding, and
for entries that rounding makes up (where the operator keeps whole matrices)."""
import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from test_gpu_pairs import product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("smallest,noise", [(2.0 ** -20, 2.0 ** -52), (2.0 ** -28, 2.0 ** -52), (2.0 ** -20, 2.0 ** -44),
                                            (2.0 ** -10, 2.0 ** -34), (2.0 ** -40, 2.0 ** -53), (2.0 ** -53, 2.0 ** -53)])
def test_single_columns(gpu, smallest, noise):
    n, n_elem = 60, 1620
    rng = np.random.default_rng(11)
    emap = np.arange(n_elem * n, dtype=np.uint32).reshape(n_elem, n)
    k = rng.choice([-1.0, 1.0], (n_elem, n, n)) * smallest ** rng.uniform(0, 1, (n_elem, n, n))
    k = np.tril(k) + np.tril(k, -1).transpose(0, 2, 1)
    ke = k + np.tril(rng.uniform(-noise, noise, (n_elem, n, n)), -1)
    ke[:, np.arange(n), np.arange(n)] = rng.uniform(1, 2, (n_elem, n))
    e = np.arange(n_elem)
    u = np.zeros((n_elem, n))
    u[e, e % n] = rng.uniform(-1, 1, n_elem)
    v = product(emap, ke, u.ravel()).reshape(n_elem, n)
    # the products of two doubles, exactly: p + q
    col, x = ke[e, :, e % n], u[e, e % n][:, None]
    ref = col.astype(np.longdouble) * x.astype(np.longdouble)
    assert np.all(np.abs(v - ref) <= 2.0 ** -44 * np.abs(ref))


@pytest.mark.parametrize("loose", [0, 1, 199, 200, 201])
def test_pairs_of_rounding(gpu, loose):
    """A chain of elements, some with a pair of entries that rounding alone makes up (200 of 1600 at most: else whole
    matrices): rows within their bound, constrained rows and columns, every way of launching the product, and a solve."""
    import torch
    n, n_elem, step = 60, 1600, 40
    rng = np.random.default_rng(loose)
    emap = (np.arange(n_elem)[:, None] * step + np.arange(n)).astype(np.uint32)
    n_dofs = int(emap.max()) + 1
    k = rng.uniform(-1, 1, (n_elem, n, n))
    ke = np.tril(k) + np.tril(k, -1).transpose(0, 2, 1) + np.tril(rng.uniform(-1, 1, (n_elem, n, n)), -1) * 2.0 ** -48
    ke[:, np.arange(n), np.arange(n)] = rng.uniform(60, 120, (n_elem, n))
    at = []
    for e in rng.permutation(n_elem)[:loose]:
        r, c = rng.choice(20, size=2, replace=False) + 20  # (rows of this element alone, in different blocks' rows)
        if (r // 2 - c // 2) % 15 == 0:
            c = 20 + (c - 20 + 2) % 20
        ke[e, r, c], ke[e, c, r] = 3.0 * 2.0 ** -50, -2.0 * 2.0 ** -50
        at.append((emap[e, r], emap[e, c]))
    fixed = np.arange(0, n_dofs, 97, dtype=np.uint64)
    maps = Maps()
    maps.set_map(n_elem, emap, n, n_dofs)
    maps.set_bdr_map(fixed, np.zeros(len(fixed)))
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_element_matrices(0, ke)
    A.finalize()
    per = (A.product_cost()[1] - 16 * n_dofs) // n_elem
    assert per == 4 * n + (22080 if loose <= 200 else 28800)
    pr = oracle.Problem(n_dofs, emap, ke, fixed, np.zeros(len(fixed)))
    size = oracle.Problem(n_dofs, emap, np.abs(ke), fixed, np.zeros(len(fixed)))
    full = torch.tensor(rng.uniform(-1, 1, n_dofs), device="cuda")
    one = torch.zeros_like(full)  # one entry of every fourth element
    one[::4 * step] = 1.0
    for a, b in at:
        one[int(b)] = 1.5
        one[int(a) // 2 * 2: int(a) // 2 * 2 + 2] = 0.0
    for u in (full, one):
        v, w = torch.empty_like(u), torch.empty_like(u)
        A.matvec_device(v.data_ptr(), u.data_ptr())
        A.synchronize()
        x = u.cpu().numpy()
        bound = size.matvec(np.abs(x))
        # (the sums of n products and of two elements add 2^-53 each; low parts 2^-47 n of the row's size)
        assert np.all(np.abs(v.cpu().numpy() - pr.matvec(x)) <= (8 * n + 14) * 2.0 ** -48 * bound)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            A.matvec_device(w.data_ptr(), u.data_ptr(), torch.cuda.current_stream().cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(v, w)
        A.set_fused_colours(1)
        A.matvec_device(w.data_ptr(), u.data_ptr())
        A.synchronize()
        A.set_fused_colours(0)
        assert torch.equal(v, w)
        A.matmult_bc_device(w.data_ptr(), u.data_ptr())
        A.synchronize()
        y = w.cpu().numpy()
        f = fixed.astype(np.int64)
        assert np.array_equal(y[f], x[f])
        keep = x.copy()
        keep[f] = 0.0
        ref = pr.matvec(keep)
        ref[f] = x[f]
        assert np.all(np.abs(y - ref) <= (8 * n + 14) * 2.0 ** -48 * (size.matvec(np.abs(keep)) + np.abs(x)))
    b = A.apply_bc(rng.standard_normal(n_dofs))
    sol, st = A.solve(b, rtol=1e-12, atol=0.0)[:2]
    assert np.linalg.norm(pr.matmult_bc(sol) - b) <= 1e-11 * np.linalg.norm(b)
    sol = A.solve_mixed(b, rtol=1e-12, inner_rtol=0.1, max_outer=40)[0]
    assert np.linalg.norm(pr.matmult_bc(sol) - b) <= 1e-11 * np.linalg.norm(b)
