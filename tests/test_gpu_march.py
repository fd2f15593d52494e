"""The marched element-coefficient operator (FP32 refinement, RG_LAYOUT_COEF) at the sizes where its
tiling changes: x-lines shorter than a 30-node strip, of a strip and one more, runs that wrap over
several lines, odd numbers of lines (two per lane in configuration 0), one plane per slab, and slabs of
several planes.  Against the oracle's paso solve; an operator that differed from A anywhere would
stall the refinement (fp64_fallback)."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu

SIZES = [(3, 2, 5), (2, 9, 4), (29, 2, 3), (30, 3, 4), (31, 4, 7), (61, 1, 6), (9, 8, 40), (59, 60, 2), (70, 41, 33),
         (29, 4), (30, 31), (31, 2), (5, 90), (250, 17)]


@pytest.mark.parametrize("cfg", [0, 1])
@pytest.mark.parametrize("ne", SIZES, ids=lambda v: "x".join(map(str, v)))
def test_marched_operator_matches_oracle(cuda, ne, cfg):
    dim, rng = len(ne), np.random.default_rng(7 + sum(ne))
    nel, nq = int(np.prod(ne)), 1 << dim
    kappa = np.exp(rng.standard_normal(nel))
    A = np.zeros((nel, dim, dim))
    for i in range(dim):
        A[:, i, i] = kappa
    Y = rng.standard_normal(nel)
    x1 = [1.0, 0.7, 1.3][:dim]  # a different spacing per axis
    d = R.Domain(dim, ne, x1)
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    elem = R.KINDS["elem"]
    R.assemble(m, rhs, keep, A=(A.reshape(-1), elem), Y=(Y, elem))
    q = np.zeros(d.n)
    q[-int(np.prod([v + 1 for v in ne[:-1]])):] = 1.0
    q[rng.integers(0, d.n, max(1, d.n // 50))] = 1.0  # scattered fixed nodes as well
    R.insert_constraint(m, rhs, R.dev(q))
    pat = O.pattern(dim, ne)
    val, rr = O.assemble(dim, ne, d.dx, pat, A=(O.EXPANDED, np.repeat(A, nq, 0).reshape(-1)),
                         Y=(O.EXPANDED, np.repeat(Y, nq)))
    O.insert_constraint(pat, val, rr, q)
    ref = O.solve_paso(pat, val, rr, tol=1e-11)
    assert ref.converged
    L.check(R.lib().rg_solver_set_config(m.h, cfg))
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10, mode=L.RG_MODE_STANDARD, precision=L.RG_PREC_FP32_REFINE,
                                       layout=L.RG_LAYOUT_COEF))
    assert st == 0 and dg.converged and dg.inner_operator == 1 and not dg.fp64_fallback
    assert np.linalg.norm(x.cpu().numpy() - ref.x) <= 1e-8 * np.linalg.norm(ref.x)


def _large(ne, seed):
    """A = kappa I on a Brick of more than 200,000 nodes, from which paso's FP64 PCG marches its operator."""
    rng = np.random.default_rng(seed)
    nel = int(np.prod(ne))
    kappa = np.exp(0.5 * rng.standard_normal(nel))
    A = np.zeros((nel, 3, 3))
    for i in range(3):
        A[:, i, i] = kappa
    Y = rng.standard_normal(nel)
    d = R.Domain(3, ne, [1.0, 0.8, 1.1])
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    R.assemble(m, rhs, keep, A=(A.reshape(-1), R.KINDS["elem"]), Y=(Y, R.KINDS["elem"]))
    q, r = np.zeros(d.n), np.zeros(d.n)
    q[: (ne[0] + 1) * (ne[1] + 1)] = 1.0
    q[rng.integers(0, d.n, d.n // 100)] = 1.0
    r[q > 0] = rng.standard_normal(int((q > 0).sum()))  # fixed values other than zero
    R.insert_constraint(m, rhs, R.dev(q), R.dev(r))
    return d, m, rhs, (A, Y, q, r)


@pytest.mark.parametrize("ne", [(61, 57, 59), (29, 201, 33), (401, 15, 31)], ids=lambda v: "x".join(map(str, v)))
def test_marched_fp64_pcg_matches_oracle(cuda, ne):
    d, m, rhs, (A, Y, q, r) = _large(ne, 3)
    assert d.n >= 200000
    pat = O.pattern(3, ne)
    val, rr = O.assemble(3, ne, d.dx, pat, A=(O.EXPANDED, np.repeat(A, 8, 0).reshape(-1)), Y=(O.EXPANDED, np.repeat(Y, 8)))
    O.insert_constraint(pat, val, rr, q, r)
    ref = O.solve_paso(pat, val, rr, tol=1e-10)
    assert ref.converged
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    for _ in range(2):
        st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10))
        assert st == 0 and dg.converged and abs(int(dg.num_iter) - ref.num_iter) <= 1
        assert np.linalg.norm(x.cpu().numpy() - ref.x) <= 1e-8 * np.linalg.norm(ref.x)


def test_values_changed_by_the_caller_are_used(cuda):
    """A caller that holds the values' address may change them: the solve then reads them."""
    import ctypes as C
    d, m, rhs, _ = _large((61, 57, 59), 4)
    p = C.c_void_p()
    L.check(R.lib().rg_matrix_values(m.h, C.byref(p)))
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    st, _ = R.solve(m, rhs, x, R.opts(tolerance=1e-10))
    assert st == 0
    d2, m2, rhs2, _ = _large((61, 57, 59), 4)
    L.check(R.lib().rg_matrix_values(m2.h, C.byref(p)))
    R._raw(p.value, d2.nnz).mul_(2.0)
    y = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    st, _ = R.solve(m2, rhs2, y, R.opts(tolerance=1e-10))
    assert st == 0 and float((y - 0.5 * x).norm() / x.norm()) <= 1e-8


def test_marched_fp64_wait_timeout_is_reported_and_recoverable(cuda):
    d, m, rhs, _ = _large((61, 57, 59), 5)
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    st, _ = R.solve(m, rhs, x, R.opts(tolerance=1e-9))
    assert st == 0
    first = x.clone()
    L.check(R.lib().rg_test_wait_limit(64, 1))
    try:
        st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-9))
    finally:
        L.check(R.lib().rg_test_wait_limit(0, 0))
    assert st == L.RG_TIMEOUT and not dg.converged
    st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-9))
    assert st == 0 and torch.equal(x, first)
