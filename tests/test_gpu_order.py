"""The order of additions is part of the results: FP64 PCG carries the rounding of its sums on, on long and badly
conditioned grids up to the solution's own error, and paso's stopping step can flip with it.  The persistent
kernels therefore add as the kernel-per-step solver (and the element-by-element assembly) did, whose results on
these systems golden/order.json records: the SHA-256 of the solution's bytes and the iterations.  So does FP32 refinement on the element coefficients, whose
products go in band order, in either configuration.  Sizes: below and
above a 32-row tile, one and several tiles per virtual block, odd node counts, pairs beyond one pass, and
an elongated Robin-like Brick on which another order ended 6e-10 away; the two largest
Bricks are where RG_LAYOUT_BAND's solves turn to the band copy."""
import hashlib
import json
import os
import sys

import numpy as np
import pytest
import torch

import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "order.json")
SIZES = [(31, 1), (30, 2), (200, 200), (255, 160), (700, 699), (1100, 1150), (1, 30, 2), (6, 5, 4), (22, 28, 114),
         (57, 54, 60), (80, 79, 82), (104, 103, 102)]
ROUTES = {"paso_csr": (L.RG_MODE_PASO, L.RG_LAYOUT_CSR), "paso_band": (L.RG_MODE_PASO, L.RG_LAYOUT_BAND),
          "textbook_csr": (L.RG_MODE_STANDARD, L.RG_LAYOUT_CSR), "textbook_band": (L.RG_MODE_STANDARD, L.RG_LAYOUT_BAND)}
REFINED = [(3, 2, 5), (29, 2, 3), (30, 3, 4), (61, 1, 6), (59, 60, 2), (70, 41, 33), (46, 101, 79), (29, 4), (30, 31),
           (250, 17)]
ASSEMBLED = [(5, 4), (64, 33), (3, 2, 5), (31, 17, 9)]


def _name(ne):
    return "x".join(map(str, ne))


def _sha(t):
    return hashlib.sha256(t.cpu().numpy().tobytes()).hexdigest()


def solve(ne, route):
    """A Robin-like problem: kappa and a reaction per element, fixed values other than zero on one face."""
    dim, rng = len(ne), np.random.default_rng(11)
    nel = int(np.prod(ne))
    A = np.zeros((nel, dim, dim))
    A[:, range(dim), range(dim)] = (0.25 + 4.0 * rng.random(nel))[:, None]
    elem = R.KINDS["elem"]
    d = R.Domain(dim, ne)
    m = R.Matrix(d)
    rhs, x = (torch.zeros(d.n, dtype=torch.float64, device="cuda") for _ in range(2))
    keep = []
    # (on the largest grid a reaction that keeps the iterations few)
    rate = 0.5 if d.n < 10 ** 6 else 2000.0
    R.assemble(m, rhs, keep, A=(A.reshape(-1), elem), D=(rate * (1.0 + rng.random(nel)), elem),
               Y=(rng.random(nel) - 0.4, elem))
    q = np.zeros(d.n)
    q[-int(np.prod([v + 1 for v in ne[:-1]])):] = 1.0
    R.insert_constraint(m, rhs, R.dev(q), R.dev(0.8 * q))
    mode, layout = ROUTES[route]
    st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-8, mode=mode, layout=layout))
    assert st == 0 and dg.converged
    return {"iterations": int(dg.num_iter), "sha256": _sha(x)}


def refine(ne, cfg=-1):
    """kappa per element, FP32 inner iterations on the element coefficients."""
    dim, rng = len(ne), np.random.default_rng(13)
    nel = int(np.prod(ne))
    A = np.zeros((nel, dim, dim))
    A[:, range(dim), range(dim)] = (0.25 + 4.0 * rng.random(nel))[:, None]
    elem = R.KINDS["elem"]
    d = R.Domain(dim, ne)
    m = R.Matrix(d)
    rhs, x = (torch.zeros(d.n, dtype=torch.float64, device="cuda") for _ in range(2))
    keep = []
    R.assemble(m, rhs, keep, A=(A.reshape(-1), elem), Y=(rng.random(nel) - 0.4, elem))
    q = np.zeros(d.n)
    q[-int(np.prod([v + 1 for v in ne[:-1]])):] = 1.0
    R.insert_constraint(m, rhs, R.dev(q), R.dev(0.8 * q))
    L.check(R.lib().rg_solver_set_config(m.h, cfg))
    st, dg = R.solve(m, rhs, x, R.opts(tolerance=1e-10, mode=L.RG_MODE_STANDARD, precision=L.RG_PREC_FP32_REFINE,
                                       layout=L.RG_LAYOUT_COEF))
    assert st == 0 and dg.converged and dg.inner_operator == 1
    return {"iterations": int(dg.num_iter), "sha256": _sha(x)}


def assemble(ne):
    """All six coefficients at the Gauss points."""
    dim, rng = len(ne), np.random.default_rng(12)
    pts = int(np.prod(ne)) << dim
    size = {"A": dim * dim, "B": dim, "C": dim, "D": 1, "X": dim, "Y": 1}
    d = R.Domain(dim, ne)
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    keep = []
    R.assemble(m, rhs, keep, **{k: (rng.random(pts * v) - 0.5, R.KINDS["exp"]) for k, v in size.items()})
    return {"values": hashlib.sha256(m.values().tobytes()).hexdigest(), "rhs": _sha(rhs)}


@pytest.fixture(scope="module")
def recorded():
    with open(GOLDEN) as f:
        return json.load(f)


@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("ne", SIZES, ids=_name)
def test_pcg_adds_in_the_order_of_a_kernel_per_step(cuda, recorded, ne, route):
    assert solve(ne, route) == recorded["solve"][route + " " + _name(ne)]


@pytest.mark.parametrize("cfg", [0, 1])
@pytest.mark.parametrize("ne", REFINED, ids=_name)
def test_refinement_adds_products_in_band_order(cuda, recorded, ne, cfg):
    assert refine(ne, cfg) == recorded["refine"][_name(ne)]


@pytest.mark.parametrize("ne", ASSEMBLED, ids=_name)
def test_assembly_adds_element_after_element(cuda, recorded, ne):
    assert assemble(ne) == recorded["assemble"][_name(ne)]


if __name__ == "__main__":  # python tests/test_gpu_order.py FILE: records what the library on PYTHONPATH returns
    with open(sys.argv[1], "w") as f:
        json.dump({"solve": {r + " " + _name(ne): solve(ne, r) for r in ROUTES for ne in SIZES},
                   "refine": {_name(ne): refine(ne) for ne in REFINED},
                   "assemble": {_name(ne): assemble(ne) for ne in ASSEMBLED}}, f, indent=1)
