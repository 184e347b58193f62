"""Host-side checks of the patch plan of the batched products: the library walks the plan on the CPU as the kernel does,
with every index checked, and the product is the oracle's; the plan of a large mesh needs no memory per thread."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from amat_gb300 import _native
from amat_gb300 import problems as P
from helpers import rel


def plan_matvec(n_dofs, emap, ke, fixed, u):
    lib = _native.libafm()
    emap = np.ascontiguousarray(emap, dtype=np.uint32)
    ke, u = np.ascontiguousarray(ke, dtype=np.float64), np.ascontiguousarray(u, dtype=np.float64)
    v, patches = np.empty(n_dofs), C.c_uint32()
    p = lambda a: C.c_void_p(a.ctypes.data)
    s = lib.afm_batched_plan_host_matvec(len(emap), n_dofs, emap.shape[1], p(emap), p(ke), p(fixed), p(u), p(v),
                                         C.byref(patches))
    assert s == 0, lib.afm_last_error().decode()
    return v, patches.value


def compare(n_dofs, emap, ke, every):
    rng = np.random.default_rng(n_dofs)
    fixed = np.zeros(n_dofs, dtype=np.uint8)
    fixed[::every] = 1
    u = rng.uniform(-1, 1, n_dofs)
    v, patches = plan_matvec(n_dofs, emap, ke, fixed, u)
    ref = oracle.Problem(n_dofs, emap, ke).matvec(np.where(fixed, 0.0, u))
    assert rel(v, ref) < 1e-14
    return patches


@pytest.mark.parametrize("kind,shape", [(P.HEX8_ELASTIC, (6, 5, 7)), (P.HEX8_ELASTIC, (8, 8, 8)), (P.HEX8_ELASTIC, (1, 1, 1)),
                                        (P.TET10_ELASTIC, (3, 2, 4)), (P.HEX20_ELASTIC, (3, 4, 2))])
def test_meshes(kind, shape):
    m = P.Mesh(kind, *shape, jitter=0.1, seed=3)
    patches = compare(m.n_dofs, m.dof_map(), m.element_matrices(ngt=3 if kind == P.HEX20_ELASTIC else 2), 13)
    if shape == (8, 8, 8):
        assert patches == 64  # 2 x 2 x 2 blocks


@pytest.mark.parametrize("n", [24, 30, 60])
def test_random_maps(n):
    rng = np.random.default_rng(n)
    emap = np.stack([rng.choice(331, size=n, replace=False) for _ in range(57)])
    compare(340, emap, rng.normal(size=(57, n, n)), 7)


def test_no_memory_per_thread():
    """64 elements among 24 million DoFs, 48 threads: a few arrays over the DoFs, not one of them for every thread."""
    code = """
import resource, sys
sys.path[:0] = %r
import numpy as np
from test_batched_plan import plan_matvec
n, n_dofs = 24, 24000001
rng = np.random.default_rng(0)
emap = np.sort(rng.choice(n_dofs, size=(64, n), replace=False), axis=1)
u, fixed = rng.uniform(-1, 1, n_dofs), np.zeros(n_dofs, dtype=np.uint8)
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
plan_matvec(n_dofs, emap, np.ones((64, n, n)), fixed, u)
print((resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before) // 1024)
""" % [os.path.dirname(os.path.abspath(__file__)), os.path.dirname(os.path.dirname(os.path.abspath(__file__)))]
    out = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, OMP_NUM_THREADS="48"), capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    # v, offsets and lists, marks and counts of the DoFs: 24 M x (8 + 8 x 4 + colouring); 48 arrays more would be 4.6 GB
    assert int(out.stdout) < 2500
