"""The FP64 band kernel (k_band64_bulk) where solves still reach it: paso's PCG with two Jacobi sweeps on
RG_LAYOUT_BAND, at ragged tiles in 3D and 2D, against the CSR kernels; and its bounded waits."""
import numpy as np
import pytest
import torch

import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _problem(ne):
    dim, rng = len(ne), np.random.default_rng(17)
    nel = int(np.prod(ne))
    A = np.zeros((nel, dim, dim))
    A[:, range(dim), range(dim)] = (0.3 + rng.random(nel))[:, None]
    elem = R.KINDS["elem"]
    d = R.Domain(dim, ne)
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    R.assemble(m, rhs, keep, A=(A.reshape(-1), elem), D=(np.full(nel, max(ne) ** 2 / 5.0), elem),
               Y=(rng.standard_normal(nel), elem))
    q = np.zeros(d.n)
    q[: int(np.prod([v + 1 for v in ne[:-1]]))] = 1.0
    R.insert_constraint(m, rhs, R.dev(q))
    return d, m, rhs


@pytest.mark.parametrize("ne", [(40, 33, 27), (7, 5, 130), (300, 211)], ids=lambda v: "x".join(map(str, v)))
def test_two_sweeps_on_the_band_copy_equal_csr(cuda, ne):
    """The condition number is below 1000 (reaction max(ne)^2 / 5), so two solves to 1e-10 agree to 1e-7."""
    d, m, rhs = _problem(ne)
    x = {}
    for layout in (L.RG_LAYOUT_CSR, L.RG_LAYOUT_BAND):
        x[layout] = torch.zeros(d.n, dtype=torch.float64, device="cuda")
        st, dg = R.solve(m, rhs, x[layout], R.opts(tolerance=1e-10, layout=layout, sweeps=2))
        assert st == 0 and dg.converged
    assert (x[L.RG_LAYOUT_BAND] - x[L.RG_LAYOUT_CSR]).norm() <= 1e-7 * x[L.RG_LAYOUT_CSR].norm()


def test_band64_wait_timeout_is_reported_and_recoverable(cuda):
    d, m, rhs = _problem((24, 20, 18))
    o = R.opts(tolerance=1e-10, layout=L.RG_LAYOUT_BAND, sweeps=2)
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    st, _ = R.solve(m, rhs, x, o)
    assert st == 0
    first = x.clone()
    L.check(R.lib().rg_test_wait_limit(64, 1))
    try:
        st, dg = R.solve(m, rhs, x, o)
    finally:
        L.check(R.lib().rg_test_wait_limit(0, 0))
    assert st == L.RG_TIMEOUT and not dg.converged and "wait" in L.last_error()
    st, dg = R.solve(m, rhs, x, o)
    assert st == 0 and dg.converged and torch.equal(x, first)
