"""The library's device memory pool: blocks that an earlier solve left full of NaN serve a later one
unchanged, and what nothing uses is bounded."""
import numpy as np
import pytest
import torch

import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _solve(ne, poison, precision, layout):
    dim = len(ne)
    d = R.Domain(dim, ne)
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    R.assemble(m, rhs, keep, A=(np.eye(dim).reshape(-1), R.KINDS["const"]), Y=(np.ones(1), R.KINDS["const"]))
    q = np.zeros(d.n)
    q[-int(np.prod([v + 1 for v in ne[:-1]])):] = 1.0
    R.insert_constraint(m, rhs, R.dev(q))
    if poison:
        rhs.fill_(float("nan"))
        R._raw(_values(m), d.nnz).fill_(float("nan"))
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-9, mode=L.RG_MODE_STANDARD, precision=precision, layout=layout))
    return st, x.clone()


def _values(m):
    import ctypes as C
    p = C.c_void_p()
    L.check(R.lib().rg_matrix_values(m.h, C.byref(p)))
    return p.value


@pytest.mark.parametrize("precision,layout", [(L.RG_PREC_FP64, L.RG_LAYOUT_CSR),
                                              (L.RG_PREC_FP32_REFINE, L.RG_LAYOUT_BAND),
                                              (L.RG_PREC_FP32_REFINE, L.RG_LAYOUT_COEF)])
def test_recycled_blocks_do_not_leak_into_a_solve(cuda, precision, layout):
    for ne in [(17, 13, 9), (60, 41)]:
        st, first = _solve(ne, False, precision, layout)
        assert st == 0
        for _ in range(2):
            assert _solve(ne, True, precision, layout)[0] != 0
        st, again = _solve(ne, False, precision, layout)
        assert st == 0 and torch.equal(first, again)


def test_unused_memory_is_bounded(cuda):
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(3):  # a pattern and values of about 3 GB
        d = R.Domain(3, (200, 200, 200))
        m = R.Matrix(d)
        torch.cuda.synchronize()
        del m, d
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free0 - (2 << 30) - (64 << 20)
