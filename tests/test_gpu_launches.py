"""A launch of a persistent solver kernel holds every SM, so it must end after a few milliseconds and let the program's
other streams have a turn: solves that take tens of milliseconds, by the library's own kernel timers.  Launches
are sized to 2 ms from an estimate of an iteration's time; three times that is allowed."""
import numpy as np
import pytest
import torch

import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu

ROUTES = {  # grid, block size, options
    "paso_csr": ((700, 699), 1, dict(tolerance=1e-8)),
    "paso_coef": ((110, 104, 108), 1, dict(tolerance=1e-9)),
    "textbook": ((600, 500), 1, dict(tolerance=1e-8, mode=L.RG_MODE_STANDARD)),
    "fp32_coef": ((150, 140, 130), 1, dict(tolerance=1e-9, mode=L.RG_MODE_STANDARD, precision=L.RG_PREC_FP32_REFINE,
                                           layout=L.RG_LAYOUT_COEF)),
    "fp32_band": ((110, 104, 108), 1, dict(tolerance=1e-9, mode=L.RG_MODE_STANDARD, precision=L.RG_PREC_FP32_REFINE,
                                           layout=L.RG_LAYOUT_BAND)),
    "system": ((200, 190), 2, dict(tolerance=1e-9)),
}


@pytest.mark.parametrize("route", ROUTES)
def test_no_launch_holds_the_gpu_for_long(cuda, route):
    ne, nb, kw = ROUTES[route]
    dim, nel = len(ne), int(np.prod(ne))
    d = R.Domain(dim, ne)
    m = R.Matrix(d, block_size=nb)
    rhs, x = (torch.zeros(d.n * nb, dtype=torch.float64, device="cuda") for _ in range(2))
    keep = []
    kappa = 0.5 + np.random.default_rng(3).random(nel)
    if nb == 1:
        A = np.zeros((nel, dim, dim))
        A[:, range(dim), range(dim)] = kappa[:, None]
        R.assemble(m, rhs, keep, A=(A.reshape(-1), R.KINDS["elem"]), Y=(np.ones(nel), R.KINDS["elem"]))
    else:
        A = np.zeros((nel, nb, dim, nb, dim))
        for i in range(nb):
            for j in range(dim):
                A[:, i, j, i, j] = kappa
        R.assemble_system(m, rhs, keep, A=(A.reshape(-1), R.KINDS["elem"]), Y=(np.ones(nel * nb), R.KINDS["elem"]))
    q = np.zeros((d.n, nb))
    q[: int(np.prod([v + 1 for v in ne[:-1]]))] = 1.0
    R.insert_constraint(m, rhs, R.dev(q.reshape(-1)))
    lib = R.lib()
    L.check(lib.rg_timers_enable(1))
    try:
        L.check(lib.rg_timers_reset())
        st, dg = R.solve(m, rhs, x, R.opts(**kw))
        torch.cuda.synchronize()
        kinds = L.timers()
    finally:
        lib.rg_timers_enable(0)
    assert st == 0 and dg.converged
    name, (launches, ms) = max(((k, (timed, total)) for k, (_, timed, total) in kinds.items()), key=lambda t: t[1][1])
    print(route, name, launches, ms)
    assert ms >= 8.0, "the solve is too short to tell"
    assert ms / launches <= 6.0, (name, launches, ms)
