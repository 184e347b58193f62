"""The work that programs have this framework do, as cases that can be timed and compared.

Every case is one call (or one solve) on an operator that a program has set up and keeps: maps, element matrices
(or node coordinates for the matrix-free operator) and boundary conditions are set, the operator is finalized, and
the vectors are on the GPU, as in a solver's iteration. The meshes are the structured ones of the example problems,
vertices jittered, element matrices by Gauss quadrature, u uniform in [-1, 1).

  op            the call
  matvec        aMatFree.matvec_device: v = K u, FP64 vectors (stored element matrices, FP64-split arithmetic)
  matmult_bc    aMatFree.matmult_bc_device: the same with boundary conditions wrapped, the product of FP64 CG
  matmult_f32   aMatFree.matmult_bc_device_f32: the FP32 product that the mixed-precision solve iterates on
  inner64       aMatFree.matvec_inner_device in symmetric inner format 4: the FP64-vector inner product
  batched       aMatFree.matvec_batched_device: nrhs right-hand sides at once, FP64
  batched_f32   the same in FP32, the product of the batched mixed solve
  free          aMatFree.matmult_bc_device of the matrix-free operator (MATFREE_TYPE::FREE), FP64
  free_f32      aMatFree.matmult_bc_device_f32 of the matrix-free operator
  cg            aMatFree.solve: Jacobi-PCG from host vectors to host vectors
  mixed         aMatFree.solve_mixed: FP32 recursion with FP64 updates, host vectors
"""
import math

import numpy as np
import torch

from amat_gb300 import MATFREE_TYPE, Maps, aMatFree
from amat_gb300 import problems as P

KINDS = {"hex8_poisson": P.HEX8_POISSON, "hex8_elastic": P.HEX8_ELASTIC, "hex20_elastic": P.HEX20_ELASTIC,
         "tet10_poisson": P.TET10_POISSON, "tet10_elastic": P.TET10_ELASTIC}
NODES = {k: P.KIND_NODES[v] for k, v in KINDS.items()}
DPN = {k: P.KIND_DPN[v] for k, v in KINDS.items()}
NGT = {"hex8_poisson": 2, "hex8_elastic": 2, "hex20_elastic": 3, "tet10_poisson": 2, "tet10_elastic": 2}
# largest meshes, in cells: about two gigabytes of element matrices at most
MOST = {"hex8_poisson": 80 ** 3, "hex8_elastic": 48 ** 3, "hex20_elastic": 42 ** 3, "tet10_poisson": 52 ** 3,
        "tet10_elastic": 24 ** 3}
# the element kinds that each call meets: batched products need more than 16 DoFs per element
OPS = {
    "matvec": ["hex8_poisson", "hex8_elastic", "hex20_elastic", "tet10_poisson", "tet10_elastic"],
    "matmult_bc": ["hex8_poisson", "hex8_elastic", "hex20_elastic", "tet10_poisson", "tet10_elastic"],
    "matmult_f32": ["hex8_poisson", "hex8_elastic", "hex20_elastic", "tet10_poisson", "tet10_elastic"],
    "inner64": ["hex8_elastic", "hex20_elastic", "tet10_elastic"],
    "batched": ["hex8_elastic", "tet10_elastic"],
    "batched_f32": ["hex8_elastic", "hex20_elastic", "tet10_elastic"],
    "free": ["hex8_elastic", "hex20_elastic", "tet10_poisson"],
    "free_f32": ["hex8_elastic", "hex20_elastic", "tet10_poisson", "tet10_elastic"],
    "cg": ["hex8_poisson"],
    "mixed": ["hex8_poisson", "tet10_poisson"],
}


def _case(op, kind, nx, ny, nz, nrhs=0, name=None):
    c = {"op": op, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "nrhs": nrhs}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest operators of a serving mix, where one product is a handful of launches
        _case("matmult_bc", "hex8_poisson", 8, 8, 8, name="poisson8_small_bc"),
        # an FP64 CG solve of the 32^3 Poisson problem, host vectors in and out: small products in a long row
        _case("cg", "hex8_poisson", 32, 32, 32, name="poisson32_cg"),
        # the product of an FP64 CG on quadratic tetrahedra
        _case("matmult_bc", "tet10_poisson", 52, 52, 52, name="tet10_poisson52_bc"),
        # the inner product of its mixed-precision solve
        _case("matmult_f32", "tet10_poisson", 47, 53, 51, name="tet10_poisson50_f32"),
        # the plain product of serendipity elasticity, the largest element matrices
        _case("matvec", "hex20_elastic", 42, 42, 42, name="hex20_42_matvec"),
        # the inner product of an ill-conditioned elastic solve (FP64 inner vectors)
        _case("inner64", "hex20_elastic", 33, 32, 31, name="hex20_32_inner64"),
        # linear bricks in elasticity, FP64 CG's product
        _case("matmult_bc", "hex8_elastic", 48, 48, 48, name="hex8_elastic48_bc"),
        # a small elastic operator's FP32 product, as served requests iterate on
        _case("matmult_f32", "hex8_elastic", 15, 13, 17, name="hex8_elastic15_f32"),
        # many load cases at once, FP32
        _case("batched_f32", "hex8_elastic", 48, 48, 48, 64, name="hex8_elastic48_rhs64_f32"),
        # ... and in FP64, the residual of the batched mixed solve
        _case("batched", "hex8_elastic", 23, 24, 25, 32, name="hex8_elastic24_rhs32"),
        # the matrix-free operator: FP64 residual product
        _case("free", "hex8_elastic", 32, 32, 32, name="hex8_elastic32_free"),
        # ... and its FP32 inner product on serendipity elements
        _case("free_f32", "hex20_elastic", 28, 27, 29, name="hex20_28_free_f32"),
    ]


def draw(rng):
    op = rng.choice(list(OPS))
    kind = rng.choice(OPS[op])
    most = MOST[kind]
    if op in ("cg", "mixed"):
        most = min(most, 30 ** 3 if kind == "hex8_poisson" else 16 ** 3)
    elif op.startswith("batched"):
        most = min(most, 24 ** 3 if kind == "hex8_elastic" else 12 ** 3)
    elif op == "free":
        most = min(most, 24 ** 3)
    cells = math.exp(rng.uniform(math.log(8 ** 3 if NODES[kind] == 8 else 5 ** 3), math.log(most)))
    # three edges around the cube root, none more than twice another
    a, b = rng.uniform(-0.3, 0.3), rng.uniform(-0.3, 0.3)
    e = cells ** (1.0 / 3.0)
    nx, ny = max(2, round(e * math.exp(a))), max(2, round(e * math.exp(b)))
    nz = max(2, min(round(cells / (nx * ny)), most // (nx * ny)))
    return _case(op, kind, nx, ny, nz, rng.choice([8, 20, 32, 48, 64]) if op.startswith("batched") else 0)


def _counts(case):
    """(elements, DoFs per element, DoFs) of a case's mesh."""
    nx, ny, nz, kind = case["nx"], case["ny"], case["nz"], case["kind"]
    vert = (nx + 1) * (ny + 1) * (nz + 1)
    if NODES[kind] == 8:
        nodes, elems = vert, nx * ny * nz
    elif NODES[kind] == 20:
        edges = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
        nodes, elems = vert + edges, nx * ny * nz
    else:
        nodes, elems = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1), 6 * nx * ny * nz
    return elems, NODES[kind] * DPN[kind], nodes * DPN[kind]


def work(case):
    """One pass: each element's symmetric matrix (or its node coordinates), its DoF map and the vectors once.
    A solve counts as thirty products, a low estimate of its iterations."""
    elems, n, dofs = _counts(case)
    op = case["op"]
    f32 = op.endswith("f32") or op == "mixed"
    entry = 4 if f32 else 8
    R = max(1, case["nrhs"])
    if op.startswith("free"):
        nodes, q = NODES[case["kind"]], NGT[case["kind"]] ** 3
        per = 3 * nodes * entry
        # Jacobian, gradient and contraction: 9, 3 dpn and 3 dpn multiply-adds per node and quadrature point
        flops = elems * q * nodes * 2 * (9 + 6 * DPN[case["kind"]])
    else:
        per = n * (n + 1) // 2 * (6 if op == "inner64" else entry)
        flops = elems * 2 * n * n * R
    times = 30 if op in ("cg", "mixed") else 1
    return {"bytes": times * (elems * (per + 4 * n) + 2 * dofs * R * entry), "flops": times * flops}


def _mesh(case, seed):
    return P.Mesh(KINDS[case["kind"]], case["nx"], case["ny"], case["nz"], jitter=0.1, seed=seed + 1)


def _vector(case, seed, dofs):
    """The pass's input vectors (host): u (dofs, or dofs x nrhs), or a load with zero boundary values."""
    rng = np.random.default_rng(seed)
    if case["op"] in ("cg", "mixed"):
        return rng.standard_normal(dofs)
    shape = (dofs, case["nrhs"]) if case["nrhs"] else (dofs,)
    f32 = case["op"].endswith("f32")
    u = rng.random(shape, dtype=np.float32 if f32 else np.float64)
    return 2.0 * u - u.dtype.type(1.0)


def prepare(case, seed):
    m = _mesh(case, seed)
    ngt = NGT[case["kind"]]
    op = case["op"]
    maps = Maps()
    maps.set_map(m.n_elem, m.dof_map(), m.ndpe, m.n_dofs)
    dofs, vals = m.boundary_conditions()
    maps.set_bdr_map(dofs, vals)
    A = aMatFree(maps)
    if op.startswith("free"):
        A.set_matfree_type(MATFREE_TYPE.FREE)
        A.set_element_kind(KINDS[case["kind"]], 1.0, 0.3, ngt)
        A.set_element_coords(0, m.coords[m.elem_nodes])
    else:
        A.set_element_matrices(0, m.element_matrices(ngt=ngt))
    A.finalize()
    if op == "inner64":
        A.set_symmetric_inner(4)
    x = _vector(case, seed, m.n_dofs)
    state = {"op": op, "A": A, "nrhs": case["nrhs"]}
    if op in ("cg", "mixed"):
        state["b"] = A.apply_bc(x)
    else:
        state["u"] = torch.from_numpy(x).cuda()
        state["v"] = torch.empty_like(state["u"])
    return state


def run(state):
    op, A = state["op"], state["A"]
    if op == "cg":
        return A.solve(state["b"], rtol=1e-12, atol=0.0)[0]
    if op == "mixed":
        return A.solve_mixed(state["b"], rtol=1e-11, max_outer=40, inner_rtol=0.1)[0]
    u, v = state["u"], state["v"]
    pv, pu = v.data_ptr(), u.data_ptr()
    if op == "matvec":
        A.matvec_device(pv, pu)
    elif op in ("matmult_bc", "free"):
        A.matmult_bc_device(pv, pu)
    elif op in ("matmult_f32", "free_f32"):
        A.matmult_bc_device_f32(pv, pu)
    elif op == "inner64":
        A.matvec_inner_device(pv, pu)
    else:
        A.matvec_batched_device(pv, pu, state["nrhs"], f32=(op == "batched_f32"))
    return v


# ---- the same in 64 bits, with plain torch -----------------------------------

_HEX = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)]
_MID = [(0, -1, -1), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (0, -1, 1), (1, 0, 1), (0, 1, 1), (-1, 0, 1),
        (-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0)]


def _hex_gradients(nodes, x):
    """Reference gradients (nodes x 3) of the 8- or 20-node brick at point x."""
    x = torch.tensor(x, dtype=torch.float64, requires_grad=True)
    N = []
    for a in range(nodes):
        if a < 8:
            p = _HEX[a]
            f = [1 + p[i] * x[i] for i in range(3)]
            n = f[0] * f[1] * f[2] / 8
            if nodes == 20:
                n = n * (p[0] * x[0] + p[1] * x[1] + p[2] * x[2] - 2)
        else:
            p = _MID[a - 8]
            n = 0.25
            for i in range(3):
                n = n * ((1 - x[i] * x[i]) if p[i] == 0 else (1 + p[i] * x[i]))
        N.append(n)
    return torch.stack([torch.autograd.grad(n, x, retain_graph=True)[0] for n in N])


def _free_product(case, xe, ue, dev):
    """Element products of linear elasticity (E = 1, nu = 0.3) integrated over bricks: (elems, n)."""
    nodes, ngt = NODES[case["kind"]], NGT[case["kind"]]
    g, w = np.polynomial.legendre.leggauss(ngt)
    lam, mu = 0.3 / (1.3 * 0.4), 0.5 / 1.3
    ue = ue.reshape(-1, nodes, 3)
    out = torch.zeros_like(ue)
    for i in range(ngt):
        for j in range(ngt):
            for k in range(ngt):
                dN = _hex_gradients(nodes, (g[i], g[j], g[k])).to(dev)
                J = torch.einsum("eai,ap->eip", xe, dN)
                G = torch.einsum("ap,epi->eai", dN, torch.linalg.inv(J))
                H = torch.einsum("eai,eaj->eij", ue, G)
                tr = H.diagonal(dim1=1, dim2=2).sum(1)
                S = mu * (H + H.transpose(1, 2)) + lam * tr[:, None, None] * torch.eye(3, device=dev, dtype=H.dtype)
                S = S * (torch.linalg.det(J) * (w[i] * w[j] * w[k]))[:, None, None]
                out += torch.einsum("eij,eaj->eai", S, G)
    return out.reshape(-1, 3 * nodes)


def exact(case, seed):
    op, kind = case["op"], case["kind"]
    if op.startswith("free") and NODES[kind] == 10:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    m = _mesh(case, seed)
    e2d = torch.from_numpy(m.dof_map().astype(np.int64)).to(dev)
    n, dofs = m.ndpe, m.n_dofs
    x = torch.from_numpy(_vector(case, seed, dofs)).to(dev).double()
    fixed = torch.zeros(dofs, dtype=torch.bool, device=dev)
    fixed[torch.from_numpy(m.boundary_conditions()[0].astype(np.int64)).to(dev)] = True
    if op.startswith("free"):
        xe = torch.from_numpy(m.coords[m.elem_nodes]).to(dev)
        u = torch.where(fixed, torch.zeros_like(x), x)
        v = torch.zeros_like(u).index_add_(0, e2d.reshape(-1), _free_product(case, xe, u[e2d], dev).reshape(-1))
        return torch.where(fixed, x, v)
    ke = torch.from_numpy(m.element_matrices(ngt=NGT[kind]))
    if op in ("cg", "mixed"):
        ke = ke.to(dev)

    def product(u):
        v = torch.zeros_like(u)
        for e0 in range(0, m.n_elem, 16384):
            d = e2d[e0:e0 + 16384]
            ve = ke[e0:e0 + 16384].to(dev) @ (u[d] if u.dim() == 2 else u[d].unsqueeze(-1))
            v.index_add_(0, d.reshape(-1), ve.reshape(-1, *u.shape[1:]))
        return v

    if op in ("matvec", "inner64", "batched", "batched_f32"):
        return product(x)
    keep = (~fixed).double()
    if op in ("matmult_bc", "matmult_f32"):
        return torch.where(fixed, x, product(x * keep))
    # Jacobi-preconditioned CG far below the solve's tolerance (zero boundary values)
    b = x * keep
    diag = torch.zeros_like(x).index_add_(0, e2d.reshape(-1), ke.diagonal(dim1=1, dim2=2).reshape(-1))
    z = b / diag
    s, r, p, rz = torch.zeros_like(b), b.clone(), z, b @ z
    for _ in range(2000):
        q = product(p) * keep
        alpha = rz / (p @ q)
        s = s + alpha * p
        r = r - alpha * q
        if r.norm() <= 1e-15 * b.norm():
            break
        z = r / diag
        rz, old = r @ z, rz
        p = z + (rz / old) * p
    return s
