"""The persistent PCG of PDE systems (block size 2 and 3) at the sizes where its tiling changes: fewer
nodes than a 4-node tile, ragged tiles, one tile per warp, tiles that stay in the shared-memory ring
and more than it holds.  Coupled elasticity-like equations with a reaction term, against the oracle's
paso solve with block Jacobi."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu

# a ring holds 2 tiles of 4 nodes per warp for blocks of 3 in 3D: 16,576 nodes on 148 SMs x 14 warps
SIZES = [(1, 1), (4, 2), (31, 30), (150, 131), (1, 1, 1), (2, 1, 4), (6, 5, 4), (13, 12, 11), (30, 29, 20)]


@pytest.mark.parametrize("nb", [2, 3])
@pytest.mark.parametrize("ne", SIZES, ids=lambda v: "x".join(map(str, v)))
def test_persistent_block_pcg_matches_oracle(cuda, ne, nb):
    dim = len(ne)
    lam, mu, eye = 1.3, 0.8, np.eye(dim)
    A = np.zeros((nb, dim, nb, dim))
    for i in range(nb):
        for j in range(dim):
            for k in range(nb):
                for l in range(dim):
                    A[i, j, k, l] = mu * (i == k) * (j == l)
                    if i < dim and k < dim:
                        A[i, j, k, l] += lam * eye[i, j] * eye[k, l] + mu * eye[i, l] * eye[j, k]
    D = (np.eye(nb) + 0.2 * (np.ones((nb, nb)) - np.eye(nb))) * max(ne) ** 2 / 5.0
    rng = np.random.default_rng(sum(ne) + nb)
    Y = rng.standard_normal((int(np.prod(ne)) * (1 << dim), nb))
    d = R.Domain(dim, ne)
    m = R.Matrix(d, nb)
    rhs = torch.zeros(d.n * nb, dtype=torch.float64, device="cuda")
    keep = []
    a, dd = A.reshape(-1, order="F"), D.reshape(-1, order="F")
    R.assemble_system(m, rhs, keep, A=(a, R.KINDS["const"]), D=(dd, R.KINDS["const"]),
                      Y=(Y.reshape(-1), R.KINDS["exp"]))
    q = np.zeros((d.n, nb))
    q[-int(np.prod([v + 1 for v in ne[:-1]])):] = 1.0
    R.insert_constraint(m, rhs, R.dev(q.reshape(-1)))
    pat = O.pattern(dim, ne)
    val, rr = O.assemble_system(dim, ne, d.dx, pat, nb, A=(O.CONSTANT, a), D=(O.CONSTANT, dd),
                                Y=(O.EXPANDED, Y.reshape(-1)))
    O.insert_constraint_block(pat, nb, val, rr, q.reshape(-1))
    ref = O.solve_paso_block(pat, nb, val, rr, tol=1e-10)
    assert ref.converged
    x = torch.zeros(d.n * nb, dtype=torch.float64, device="cuda")
    for _ in range(2):  # the second solve starts from what the first one left behind
        st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10))
        assert st == 0 and dg.converged and abs(int(dg.num_iter) - ref.num_iter) <= 1
        assert np.linalg.norm(x.cpu().numpy() - ref.x) <= 1e-8 * np.linalg.norm(ref.x)


def test_block_pcg_wait_timeout_is_reported_and_recoverable(cuda):
    """Posts and copies withheld, so that the bounded waits run out: RG_TIMEOUT, and the next solve on
    the same matrix is unchanged."""
    d = R.Domain(2, (20, 17))
    m = R.Matrix(d, 2)
    rhs = torch.zeros(d.n * 2, dtype=torch.float64, device="cuda")
    keep = []
    A = np.einsum("ik,jl->ijkl", np.eye(2), np.eye(2))
    R.assemble_system(m, rhs, keep, A=(A.reshape(-1, order="F"), R.KINDS["const"]),
                      D=(np.eye(2).reshape(-1), R.KINDS["const"]), Y=(np.ones(2), R.KINDS["const"]))
    x = torch.zeros_like(rhs)
    st, _ = R.solve(m, rhs, x, R.opts(tolerance=1e-10))
    assert st == 0
    first = x.clone()
    L.check(R.lib().rg_test_wait_limit(64, 1))
    try:
        st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10))
    finally:
        L.check(R.lib().rg_test_wait_limit(0, 0))
    assert st == L.RG_TIMEOUT and "wait" in L.last_error() and not dg.converged
    st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10))
    assert st == 0 and torch.equal(x, first)
