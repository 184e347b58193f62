"""Products of one operator on several streams, and its solves, run in turn: they share buffers of the operator. A
product still pending on a caller's stream ends before a solve that follows it returns, also where the solve's FP64
products go another way than its captured FP32 iterations, and keeps its bits."""
import ctypes as C

import numpy as np
import pytest

import oracle
from amat_gb300 import PRECISION, Maps, aMatFree
from helpers import rel

pytestmark = pytest.mark.gpu


def chain(n, n_elem):
    """A row of symmetric, diagonally dominant elements that share a third of their DoFs (two colours)."""
    rng = np.random.default_rng(n)
    step = n - n // 3
    emap = (np.arange(n_elem)[:, None] * step + np.arange(n)).astype(np.uint32)
    k = rng.uniform(-1, 1, (n_elem, n, n))
    ke = k + k.transpose(0, 2, 1)
    ke[:, np.arange(n), np.arange(n)] = 2.0 * n + rng.uniform(0, n, (n_elem, n))
    n_dofs = int(emap.max()) + 1
    maps = Maps()
    maps.set_map(n_elem, emap, n, n_dofs)
    A = aMatFree(maps)
    A.set_precision(PRECISION.FP64_SPLIT)
    A.set_element_matrices(0, ke)
    A.finalize()
    return emap, ke, n_dofs, A


def pending(torch, caller, call, refs, count):
    """`count` products behind a wait of some milliseconds on the caller's stream, checked by the returned function."""
    outs = [torch.full_like(refs, float("nan")) for _ in range(count)]
    torch.cuda.synchronize()
    with torch.cuda.stream(caller):
        torch.cuda._sleep(20_000_000)
    for o in outs:
        call(o.data_ptr(), caller.cuda_stream)

    def check():
        done = caller.query()
        caller.synchronize()
        assert done
        for o in outs:
            assert torch.equal(o, refs)
    return check


# n = 36: the FP64 product of 5600 elements or more per colour runs per colour, the FP32 one on the shared buffer
@pytest.mark.parametrize("n,n_elem", [(36, 12000), (36, 500), (60, 2000), (10, 4000)])
def test_mixed_solve_after_a_pending_product(gpu, n, n_elem):
    import torch
    emap, ke, n_dofs, A = chain(n, n_elem)
    rng = np.random.default_rng(1)
    b = rng.standard_normal(n_dofs)
    first = A.solve_mixed(b, rtol=1e-10)[0]  # (captures the iterations)
    u = torch.tensor(rng.uniform(-1, 1, n_dofs), device="cuda", dtype=torch.float32)
    ref = torch.empty_like(u)
    A.matvec_device_f32(ref.data_ptr(), u.data_ptr())
    A.synchronize()
    check = pending(torch, torch.cuda.Stream(), lambda v, s: A.matvec_device_f32(v, u.data_ptr(), s), ref, 20)
    x = A.solve_mixed(b, rtol=1e-10)[0]
    check()
    assert np.array_equal(x, first)
    assert rel(oracle.Problem(n_dofs, emap, ke).matvec(x), b) < 1e-9


@pytest.mark.parametrize("mixed", [False, True])
def test_batched_solve_after_a_pending_product(gpu, mixed):
    """hex20-sized elements: the FP64 residual takes the launches per colour, the FP32 iterations may take the patches."""
    import torch
    emap, ke, n_dofs, A = chain(60, 800)
    nrhs = 16
    rng = np.random.default_rng(2)
    B = torch.tensor(rng.standard_normal((n_dofs, nrhs)), device="cuda")

    def solve():
        X = torch.zeros_like(B)
        torch.cuda.current_stream().synchronize()
        A.solve_batched_device(B.data_ptr(), X.data_ptr(), nrhs, rtol=1e-10, mixed=mixed)
        return X
    first = solve()
    U = torch.tensor(rng.uniform(-1, 1, (n_dofs, nrhs)), device="cuda", dtype=torch.float32)
    ref = torch.empty_like(U)
    A.matvec_batched_device(ref.data_ptr(), U.data_ptr(), nrhs, f32=True)
    A.synchronize()
    check = pending(torch, torch.cuda.Stream(),
                    lambda v, s: A.matvec_batched_device(v, U.data_ptr(), nrhs, f32=True, stream=s), ref, 20)
    X = solve()
    check()
    assert torch.equal(X, first)


def cudart():
    for name in ("libcudart.so.13", "/usr/local/cuda/lib64/libcudart.so"):
        try:
            return C.CDLL(name)
        except OSError:
            continue
    pytest.skip("no shared CUDA runtime")


def test_streams_that_come_and_go(gpu):
    """A stream made after another was destroyed may have its handle: its product still waits for the one before."""
    import torch
    emap, ke, n_dofs, A = chain(24, 3000)
    rt = cudart()
    us = [torch.tensor(np.random.default_rng(k).uniform(-1, 1, n_dofs), device="cuda") for k in range(2)]
    refs = []
    for x in us:
        v = torch.empty_like(x)
        A.matvec_device(v.data_ptr(), x.data_ptr())
        A.synchronize()
        refs.append(v)
    outs = [torch.empty_like(us[0]) for _ in range(40)]
    torch.cuda.synchronize()
    for k, o in enumerate(outs):
        s = C.c_void_p()
        assert rt.cudaStreamCreateWithFlags(C.byref(s), 1) == 0
        A.matvec_device(o.data_ptr(), us[k % 2].data_ptr(), s.value)
        assert rt.cudaStreamDestroy(s) == 0
    A.synchronize()
    torch.cuda.synchronize()
    for k, o in enumerate(outs):
        assert torch.equal(o, refs[k % 2])


@pytest.mark.parametrize("again", [False, True])
@pytest.mark.parametrize("n", [10, 24])
def test_product_pending_at_the_end(gpu, n, again):
    """An operator is finalized again or destroyed while a product waits on a caller's stream: its memory is given back
    after the product, so that what other operators put there in the meantime is not read."""
    import torch
    emap, ke, n_dofs, A = chain(n, 3000)
    u = torch.tensor(np.random.default_rng(n).uniform(-1, 1, n_dofs), device="cuda")
    ref, v = torch.empty_like(u), torch.empty_like(u)
    A.matvec_device(ref.data_ptr(), u.data_ptr())
    A.synchronize()
    caller = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(caller):
        torch.cuda._sleep(100_000_000)
    A.matvec_device(v.data_ptr(), u.data_ptr(), caller.cuda_stream)
    if again:
        A.set_element_matrices(0, 2.0 * ke)
        A.finalize()
    else:
        A.close()
    other = chain(n, 3000 + n)[3]
    other.synchronize()
    torch.cuda.synchronize()
    assert torch.equal(v, ref)


@pytest.mark.parametrize("n", [24, 60])
def test_recorded_product_beside_others(gpu, n):
    """A recorded product has u scales of its own: replayed beside products of u of another size, it keeps its bits."""
    import torch
    emap, ke, n_dofs, A = chain(n, 300)
    rng = np.random.default_rng(n)
    u = torch.tensor(rng.uniform(-1, 1, n_dofs), device="cuda")
    big = u * 2.0 ** 200
    v, w, ref = torch.empty_like(u), torch.empty_like(u), torch.empty_like(u)
    A.matvec_device(ref.data_ptr(), u.data_ptr())
    A.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.matvec_device(v.data_ptr(), u.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for _ in range(50):
        v.fill_(float("nan"))
        torch.cuda.synchronize()
        g.replay()
        A.matvec_device(w.data_ptr(), big.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(v, ref)
        assert torch.equal(w, ref * 2.0 ** 200)
