"""Device memory: what a program destroys goes back to the device, addresses that the library hands out are ordinary
allocations, destroying a matrix leaves another thread's capture alone, and the arrays a domain keeps for its next
matrix of the same block size carry nothing over."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _poisson(ne):
    d = R.Domain(len(ne), ne)
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    R.assemble(m, rhs, keep, A=(np.eye(len(ne)).reshape(-1), R.KINDS["const"]), Y=(np.ones(1), R.KINDS["const"]))
    q = np.zeros(d.n)
    q[: int(np.prod([v + 1 for v in ne[:-1]]))] = 1.0
    R.insert_constraint(m, rhs, R.dev(q))
    return d, m, rhs


def test_destroyed_objects_give_their_memory_back(cuda):
    """60 Bricks of 48^3 with a solve each, about 50 MB a piece in blocks of up to 24 MB, alive together: after the
    last is gone less than 64 MB are missing."""
    d, m, rhs = _poisson((48, 48, 48))  # (kernels are loaded)
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    assert R.solve(m, rhs, x, R.opts(tolerance=1e-2))[0] == 0
    del d, m, rhs, x
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    alive = []
    for _ in range(60):
        d, m, rhs = _poisson((48, 48, 48))
        x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
        assert R.solve(m, rhs, x, R.opts(tolerance=1e-2))[0] == 0
        alive.append((m, d))
    del d, m, rhs, x
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert torch.cuda.mem_get_info()[0] < free0 - (2 << 30)
    alive.clear()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free0 - (64 << 20)


def test_values_can_be_shared_between_processes(cuda):
    """cudaIpcGetMemHandle takes the address that rg_matrix_values returns, on small matrices too."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    d, m, _ = _poisson((20, 10))
    p = C.c_void_p()
    L.check(R.lib().rg_matrix_values(m.h, C.byref(p)))
    err, _handle = rt.cudaIpcGetMemHandle(p.value)
    assert err == rt.cudaError_t.cudaSuccess, err


def test_destroying_a_matrix_leaves_another_threads_capture_alone(cuda):
    stream = torch.cuda.Stream()
    x = torch.zeros(1024, device="cuda")
    torch.cuda.synchronize()
    began, done, failed = threading.Event(), threading.Event(), []
    d, m, _ = _poisson((30, 20))
    holder = [d, m]

    def destroy():
        try:
            torch.cuda.set_device(0)
            began.wait(30)
            holder.clear()
        except Exception as e:  # noqa: BLE001
            failed.append(e)
        finally:
            done.set()

    del d, m
    t = threading.Thread(target=destroy)
    t.start()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
        x += 1.0
        began.set()
        assert done.wait(60)
        x += 1.0
    t.join()
    assert not failed
    g.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 2.0


def test_a_systems_arrays_serve_the_next_matrix(cuda):
    """The same 2D system solved on fresh matrices of one domain, with NaN left in the arrays in between."""
    ne, nb = (33, 21), 2
    rng = np.random.default_rng(5)
    nel = int(np.prod(ne))
    A = np.zeros((nel, 2, 2, 2, 2))
    for i in range(2):
        for j in range(2):
            A[:, i, j, i, j] = 0.5 + rng.random(nel)
    Y = rng.random((nel, 2))
    d = R.Domain(2, ne)

    def once(poison):
        m = R.Matrix(d, block_size=nb)
        rhs, x = (torch.zeros(d.n * nb, dtype=torch.float64, device="cuda") for _ in range(2))
        keep = []
        R.assemble_system(m, rhs, keep, A=(A.reshape(-1), R.KINDS["elem"]), Y=(Y.reshape(-1), R.KINDS["elem"]))
        q = np.zeros((d.n, nb))
        q[: ne[0] + 1] = 1.0
        R.insert_constraint(m, rhs, R.dev(q.reshape(-1)))
        if poison:
            rhs.fill_(float("nan"))
        st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-9))
        if poison:
            p = C.c_void_p()
            L.check(R.lib().rg_matrix_values(m.h, C.byref(p)))
            R._raw(p.value, d.nnz * nb * nb).fill_(float("nan"))
            torch.cuda.synchronize()
        return st, x

    st, first = once(False)
    assert st == 0
    assert once(True)[0] != 0
    st, again = once(False)
    assert st == 0 and torch.equal(first, again)
