"""The persistent FP64 PCG (paso with residual smoothing, and textbook) at the sizes where its
tiling changes: fewer rows than a 32-row tile, ragged last tiles, one tile per warp, tiles that
stay in the shared-memory ring, and more tiles than the ring holds.  A = kappa I with a reaction
term, against the oracle's paso solve of the same system."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu

# a ring holds 2 x 32 rows per warp in 3D (151,552 rows on 148 SMs x 16 warps), 6 x 32 in 2D (454,656)
SIZES = [(1, 1), (31, 1), (30, 2), (255, 160), (700, 699), (1, 1, 1), (1, 30, 2), (6, 5, 4), (31, 31, 3),
         (57, 54, 50)]


@pytest.mark.parametrize("mode", [L.RG_MODE_PASO, L.RG_MODE_STANDARD])
@pytest.mark.parametrize("ne", SIZES, ids=lambda v: "x".join(map(str, v)))
def test_persistent_pcg_matches_oracle(cuda, ne, mode):
    dim, rng = len(ne), np.random.default_rng(sum(ne))
    nel = int(np.prod(ne))
    kappa = np.exp(0.5 * rng.standard_normal(nel))
    A = np.zeros((nel, dim, dim))
    for i in range(dim):
        A[:, i, i] = kappa
    Dc = np.full(nel, max(ne) ** 2 / 5.0)
    Y = rng.standard_normal(nel)
    d = R.Domain(dim, ne)
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    elem = R.KINDS["elem"]
    R.assemble(m, rhs, keep, A=(A.reshape(-1), elem), D=(Dc, elem), Y=(Y, elem))
    q = np.zeros(d.n)
    q[-int(np.prod([v + 1 for v in ne[:-1]])):] = 1.0
    R.insert_constraint(m, rhs, R.dev(q))
    nq = 1 << dim
    pat = O.pattern(dim, ne)
    val, rr = O.assemble(dim, ne, d.dx, pat, A=(O.EXPANDED, np.repeat(A, nq, 0).reshape(-1)),
                         D=(O.EXPANDED, np.repeat(Dc, nq)), Y=(O.EXPANDED, np.repeat(Y, nq)))
    O.insert_constraint(pat, val, rr, q)
    ref = O.solve_paso(pat, val, rr, tol=1e-10)
    assert ref.converged
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    for _ in range(2):  # the second solve starts from what the first one left behind
        st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10, mode=mode))
        assert st == 0 and dg.converged
        assert np.linalg.norm(x.cpu().numpy() - ref.x) <= 1e-8 * np.linalg.norm(ref.x)
        if mode == L.RG_MODE_PASO:
            assert abs(int(dg.num_iter) - ref.num_iter) <= 1


def test_persistent_pcg_stops_at_iter_max(cuda):
    """iter_max reached inside a launch: RG_MAXITER with the paso count, as the reference."""
    ne = (40, 33)
    d = R.Domain(2, ne)
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    R.assemble(m, rhs, keep, A=(np.eye(2).reshape(-1), R.KINDS["const"]), Y=(np.ones(1), R.KINDS["const"]))
    q = np.zeros(d.n)
    q[: ne[0] + 1] = 1.0
    R.insert_constraint(m, rhs, R.dev(q))
    x = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    for mode in (L.RG_MODE_PASO, L.RG_MODE_STANDARD):
        st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10, mode=mode, iter_max=7))
        assert st == L.RG_MAXITER and not dg.converged and 6 <= int(dg.num_iter) <= 9


def test_textbook_band_route_on_large_grids(cuda):
    """RG_LAYOUT_BAND's textbook PCG runs on the band copy from 1.5 million rows of a 3D grid: the same
    solution as on the CSR values.  The balanced matrix's condition number is below 1000 (reaction
    max(ne)^2 / 5 against 12 max(ne)^2 kappa), so two solves to 1e-10 agree to 1e-7."""
    ne = (120, 115, 108)
    rng = np.random.default_rng(8)
    nel = int(np.prod(ne))
    A = np.zeros((nel, 3, 3))
    A[:, range(3), range(3)] = np.exp(0.3 * rng.standard_normal(nel))[:, None]
    elem = R.KINDS["elem"]
    d = R.Domain(3, ne)
    m = R.Matrix(d)
    assert d.n >= 1500000
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    R.assemble(m, rhs, keep, A=(A.reshape(-1), elem), D=(np.full(nel, max(ne) ** 2 / 5.0), elem),
               Y=(rng.standard_normal(nel), elem))
    x = {}
    for layout in (L.RG_LAYOUT_BAND, L.RG_LAYOUT_CSR):
        x[layout] = torch.zeros(d.n, dtype=torch.float64, device="cuda")
        st, dg = R.solve(m, rhs, x[layout], R.opts(tolerance=1e-10, mode=L.RG_MODE_STANDARD, layout=layout))
        assert st == 0 and dg.converged
    assert (x[L.RG_LAYOUT_BAND] - x[L.RG_LAYOUT_CSR]).norm() <= 1e-7 * x[L.RG_LAYOUT_CSR].norm()
