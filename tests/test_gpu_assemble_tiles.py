"""Interior assembly at the edges of its tiling: rows per warp (31) and per block (124), x-lines shorter
than a warp, rows that cross the ends of lines and planes; coefficients at the Gauss points mixed with
per-element and constant ones, absent ones, and arrays off a 16-byte boundary.  Against the oracle:
values and right hand side to 1e-13 of the row's largest entry (sums of at most 8 elements x 8 points)."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import oracle as O
import rgcapi as R
from esys_b200 import _lib as L

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (2, 3, 9), (30, 1, 2), (31, 3, 2), (13, 4, 3), (61, 2, 2), (1, 1), (29, 3), (30, 2), (32, 5), (3, 70)]
# kind of A, B, C, D, X, Y: e = at the Gauss points, p = per element, c = constant, - = absent
KINDS = ["eeeeee", "e-p-ec", "-epcpe", "c--e--", "p-pcep", "e----e", "----ee"]


def _shapes(dim):
    return {"A": (dim, dim), "B": (dim,), "C": (dim,), "D": (), "X": (dim,), "Y": ()}


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("kinds", KINDS)
@pytest.mark.parametrize("ne", SIZES, ids=lambda v: "x".join(map(str, v)))
def test_assembly_tiles_match_oracle(cuda, ne, kinds, shift):
    dim, nel = len(ne), int(np.prod(ne))
    nq, rng = 1 << dim, np.random.default_rng(sum(ne) + 100 * KINDS.index(kinds))
    d = R.Domain(dim, ne, [1.0, 0.6, 1.7][:dim])
    m = R.Matrix(d)
    rhs = torch.zeros(d.n, dtype=torch.float64, device="cuda")
    cs, ref, keep = [], {}, []
    for name, k in zip("ABCDXY", kinds):
        if k == "-":
            cs.append(L.rg_coef(None, L.RG_COEF_EMPTY))
            continue
        lead = {"e": (nel, nq), "p": (nel,), "c": (1,)}[k]
        v = rng.standard_normal(lead + _shapes(dim)[name])
        t = torch.zeros(v.size + 2, dtype=torch.float64, device="cuda")
        t[shift:shift + v.size] = torch.from_numpy(v.reshape(-1)).cuda()
        keep.append(t)
        kind = {"e": L.RG_COEF_EXPANDED, "p": L.RG_COEF_PER_ELEMENT, "c": L.RG_COEF_CONSTANT}[k]
        cs.append(L.rg_coef(t.data_ptr() + 8 * shift, kind))
        full = np.broadcast_to(v if k == "e" else (v[:, None] if k == "p" else v[:, None]),
                               (nel, nq) + _shapes(dim)[name])
        ref["C_" if name == "C" else name] = (O.EXPANDED, np.ascontiguousarray(full).reshape(-1))
    L.set_stream_from_torch()
    L.check(R.lib().rg_assemble_single(m.h, R.ptr(rhs), *[C.byref(c) for c in cs]))
    pat = O.pattern(dim, ne)
    val, rr = O.assemble(dim, ne, d.dx, pat, **ref)
    got, ptr = m.values(), np.asarray(pat.ptr)
    scale = np.repeat(np.maximum.reduceat(np.abs(val), ptr[:-1]), np.diff(ptr)) if np.abs(val).max() > 0 else 1.0
    assert np.all(np.abs(got - val) <= 1e-13 * np.maximum(scale, np.abs(val).max() * 1e-3))
    assert np.abs(rhs.cpu().numpy() - rr).max() <= 1e-13 * max(np.abs(rr).max(), 1e-300)
