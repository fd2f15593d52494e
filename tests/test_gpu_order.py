"""The order of additions is part of the results: conjugate gradients carry rounding on.  Assembly adds element
after element, as one thread per row did, whose values golden/order.json records (SHA-256 of their bytes)."""
import hashlib
import json
import os
import sys

import numpy as np
import pytest
import torch

import rgcapi as R

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "order.json")
ASSEMBLED = [(5, 4), (64, 33), (3, 2, 5), (31, 17, 9)]


def _name(ne):
    return "x".join(map(str, ne))


def _sha(t):
    return hashlib.sha256(t.cpu().numpy().tobytes()).hexdigest()


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


@pytest.mark.parametrize("ne", ASSEMBLED, ids=_name)
def test_assembly_adds_element_after_element(cuda, recorded, ne):
    assert assemble(ne) == recorded["assemble"][_name(ne)]


if __name__ == "__main__":  # python tests/test_gpu_order.py FILE: records what the library on PYTHONPATH returns
    with open(sys.argv[1], "w") as f:
        json.dump({"assemble": {_name(ne): assemble(ne) for ne in ASSEMBLED}}, f, indent=1)
