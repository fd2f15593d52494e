"""The work that programs built on this library have it do, as cases that can be timed and compared.

Each case goes through the public entry points (the escript mirror, the C ABI through its ctypes
loader, the batch and warm-start modules) on seeded synthetic inputs on the GPU.  `listed` names the
cases, `draw` gives more of the same ranges, `prepare` makes what a program holds before the call,
`run` is one pass, `work` what a pass cannot do without, `exact` the result in 64 bits from plain torch.
"""
import ctypes as C
import itertools
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "esys-escript.github.io_b200"))

F64 = torch.float64
DEV = "cuda"


def listed():
    return [
        # a script's first solve: Poisson on a 200 x 200 Rectangle with the default options (paso PCG +
        # Jacobi in FP64 on the CSR matrix, tolerance 1e-8); the coefficients change every pass, as in a
        # parameter study, so the operator is rebuilt
        {"name": "rect200_poisson", "kind": "pde", "ne": "200x200", "terms": "poisson", "tol": 1e-8},
        # the smallest calls: a ragged little Brick with reaction, Robin faces and a non-zero Dirichlet value
        {"name": "brick_small_robin", "kind": "pde", "ne": "21x17x14", "terms": "robin", "tol": 1e-8},
        # the reference's own workload: Brick 128^3, variable kappa at the Gauss points, default options
        {"name": "brick128_poisson", "kind": "pde", "ne": "128x128x128", "terms": "poisson", "tol": 1e-8},
        # time stepping: the operator stays, every step brings a new source; textbook PCG on the band copy
        {"name": "heat_steps_2d", "kind": "steps", "ne": "403x297", "tol": 1e-8},
        # FP32 inner / FP64 refinement with the operator from the element coefficients (C ABI, A per element)
        {"name": "brick128_refine", "kind": "refine", "ne": "128x128x128", "corr": 8.0, "tol": 1e-10},
        # the largest: the same on 256^3 (16.9 million unknowns)
        {"name": "brick256_refine", "kind": "refine", "ne": "256x256x256", "corr": 16.0, "tol": 1e-10},
        # FP32 refinement where the operator is not kappa I: anisotropic A and a reaction term (band copy)
        {"name": "aniso_refine", "kind": "aniso", "ne": "95x112x81", "tol": 1e-10},
        # the learned warm start: network guess, smoothing, then FP32 refinement on a 64^3 Brick
        {"name": "learned64", "kind": "learned", "edge": 64, "corr": 8.0, "tol": 1e-10},
        # many systems of uneven size with 8 right hand sides each, solved together
        {"name": "batch12x8", "kind": "batch", "systems": 12, "nrhs": 8, "pick": 7, "lo": 32, "hi": 96, "tol": 1e-10},
        # linear elasticity: three equations, Lame coefficients at the Gauss points, default options
        {"name": "elastic3d", "kind": "elastic", "ne": "36x31x28", "tol": 1e-8},
        # assembly alone: every coefficient of the general PDE at the Gauss points, then the constraint
        {"name": "assemble96", "kind": "assemble", "ne": "96x97x95", "coefs": "ABCDXY", "layout": "expanded"},
        # training of the warm-start network: one decoder convolution, forward and backward (bf16)
        {"name": "conv_dec0a", "kind": "conv", "n": 4, "grid": "64x64x64", "cin": 48, "cout": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pde", "pde", "pde", "steps", "refine", "refine", "aniso", "learned", "batch", "elastic",
                       "assemble", "conv"])
    three = lambda lo, hi: "x".join(str(_log(rng, lo, hi)) for _ in range(3))  # noqa: E731
    if kind == "pde":
        if rng.random() < 0.4:
            ne = "%dx%d" % (_log(rng, 20, 700), _log(rng, 20, 700))
        else:
            ne = three(8, 128)
        return {"kind": kind, "ne": ne, "terms": rng.choice(["poisson", "robin"]), "tol": 1e-8}
    if kind == "steps":
        ne = "%dx%d" % (_log(rng, 40, 900), _log(rng, 40, 900)) if rng.random() < 0.6 else three(12, 96)
        return {"kind": kind, "ne": ne, "tol": 1e-8}
    if kind == "refine":
        return {"kind": kind, "ne": three(24, 200), "corr": round(rng.uniform(4.0, 16.0), 2), "tol": 1e-10}
    if kind == "aniso":
        return {"kind": kind, "ne": three(20, 128), "tol": 1e-10}
    if kind == "learned":
        return {"kind": kind, "edge": rng.choice([64, 128]), "corr": round(rng.uniform(4.0, 12.0), 2),
                "tol": 1e-10}
    if kind == "batch":
        return {"kind": kind, "systems": rng.randint(2, 14), "nrhs": rng.choice([1, 2, 4, 8, 8]),
                "pick": rng.randrange(10 ** 6), "lo": 20, "hi": rng.randint(40, 96), "tol": 1e-10}
    if kind == "elastic":
        ne = "%dx%d" % (_log(rng, 12, 160), _log(rng, 12, 160)) if rng.random() < 0.35 else three(7, 40)
        return {"kind": kind, "ne": ne, "tol": 1e-8}
    if kind == "assemble":
        coefs = rng.choice(["AY", "ADY", "ABCDXY", "ADXY", "ACY"])
        if rng.random() < 0.3:
            ne = "%dx%d" % (_log(rng, 60, 1200), _log(rng, 60, 1200))
        else:
            ne = three(16, 128)
        return {"kind": kind, "ne": ne, "coefs": coefs, "layout": rng.choice(["expanded", "element"])}
    cin, cout = rng.choice([(16, 16), (16, 32), (32, 32), (48, 16), (80, 32), (32, 48), (48, 48), (112, 48)])
    g = rng.choice([16, 32, 64])
    return {"kind": "conv", "n": rng.randint(1, 8), "grid": "%dx%dx%d" % (g, g, rng.choice([16, 32, 64])),
            "cin": cin, "cout": cout}


# ---------------------------------------------------------------------------------------------- inputs

def _ints(text):
    return tuple(int(v) for v in text.split("x"))


def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt * 7919 + 11) % (1 << 62))


def _field(ne, corr, gen):
    """A zero-mean, unit-variance Gaussian random field per element, periodic, correlation `corr` cells;
    ne = (nx, ny[, nz]), the result has x fastest."""
    shape = tuple(reversed(ne))
    noise = torch.randn(shape, generator=gen, device=DEV, dtype=F64)
    k2 = 0.0
    for ax, cnt in enumerate(shape):
        f = torch.fft.fftfreq(cnt, device=DEV, dtype=F64) * (2 * math.pi)
        k2 = k2 + (f ** 2).reshape([-1 if a == ax else 1 for a in range(len(shape))])
    g = torch.fft.ifftn(torch.fft.fftn(noise) * torch.exp(-0.5 * corr ** 2 * k2)).real
    g = g - g.mean()
    return g / g.std().clamp_min(1e-6)


def _blobs(ne, gen, count=4, width=3.0):
    """Sum of Gaussian blobs `width` cells wide at the element centres, amplitudes U(-1, 1)."""
    d = len(ne)
    amp = torch.rand(count, generator=gen, device=DEV, dtype=F64) * 2 - 1
    ctr = torch.rand((count, d), generator=gen, device=DEV, dtype=F64)
    y = torch.zeros(tuple(reversed(ne)), device=DEV, dtype=F64)
    for b in range(count):
        f = amp[b]
        for ax in range(d):
            x = (torch.arange(ne[ax], device=DEV, dtype=F64) + 0.5) / ne[ax]
            g = torch.exp(-(x - ctr[b, ax]) ** 2 / (2 * (width / ne[ax]) ** 2))
            f = f * g.reshape([-1 if a == d - 1 - ax else 1 for a in range(d)])
        y = y + f
    return y


def _top(ne):
    """1 on the nodes of the last face of the last axis."""
    nn = [v + 1 for v in ne]
    q = torch.zeros(tuple(reversed(nn)), device=DEV, dtype=F64)
    q[-1] = 1.0
    return q.reshape(-1)


def _pde_inputs(case, seed):
    """Per-element kappa, source, and the Robin case's further coefficients."""
    ne = _ints(case["ne"])
    gen = _gen(seed)
    out = {"kappa": torch.exp(_field(ne, 8.0, gen)).reshape(-1), "y": _blobs(ne, gen).reshape(-1)}
    if case.get("terms") == "robin":
        out["d"] = 0.5 + torch.rand(out["kappa"].numel(), generator=gen, device=DEV, dtype=F64)
        out["flux"] = float(torch.rand((), generator=gen, device=DEV)) - 0.5
        out["value"] = float(torch.rand((), generator=gen, device=DEV)) + 0.5
    return out


def _batch_shapes(case):
    rng = torch.Generator().manual_seed(case["pick"])
    e = torch.randint(case["lo"], case["hi"] + 1, (case["systems"], 3), generator=rng)
    return [tuple(int(v) for v in row) for row in e]


def _lame(case, seed):
    ne = _ints(case["ne"])
    gen = _gen(seed)
    mu = torch.exp(0.5 * _field(ne, 6.0, gen)).reshape(-1)
    lam = torch.exp(0.5 * _field(ne, 6.0, gen)).reshape(-1)
    load = torch.stack([_blobs(ne, gen).reshape(-1) for _ in ne], 1)
    return mu, lam, load


def _lame_tensor(mu, lam, d):
    """A[e, i, j, k, l] = lam delta_ij delta_kl + mu (delta_ik delta_jl + delta_il delta_jk)."""
    eye = torch.eye(d, device=DEV, dtype=F64)
    a = torch.einsum("ij,kl->ijkl", eye, eye)
    b = torch.einsum("ik,jl->ijkl", eye, eye) + torch.einsum("il,jk->ijkl", eye, eye)
    return lam[:, None, None, None, None] * a + mu[:, None, None, None, None] * b


def _aniso(case, seed):
    """Symmetric positive definite A per element (column-major data points), D and Y per element."""
    ne = _ints(case["ne"])
    gen = _gen(seed)
    k = torch.exp(0.7 * _field(ne, 8.0, gen)).reshape(-1)
    b = torch.randn((k.numel(), 3, 3), generator=gen, device=DEV, dtype=F64) * 0.3
    a = k[:, None, None] * (torch.eye(3, device=DEV, dtype=F64) + torch.einsum("eij,ekj->eik", b, b))
    dd = 10.0 * torch.rand(k.numel(), generator=gen, device=DEV, dtype=F64)
    return a, dd, _blobs(ne, gen).reshape(-1)


def _assembly_inputs(case, seed):
    """Coefficient arrays in escript's layout: (elements[, points], comps), A with j before i."""
    ne = _ints(case["ne"])
    d = len(ne)
    gen = _gen(seed)
    lead = (math.prod(ne),) + ((1 << d,) if case["layout"] == "expanded" else ())
    comp = {"A": (d, d), "B": (d,), "C": (d,), "D": (), "X": (d,), "Y": ()}
    return {c: torch.randn(lead + comp[c], generator=gen, device=DEV, dtype=F64) for c in case["coefs"]}


def _conv_inputs(case, seed):
    """bf16 activations after a ReLU, weights, and an output gradient after its ReLU mask."""
    n, (w, h, d) = case["n"], _ints(case["grid"])
    gen = _gen(seed)
    x = torch.zeros((n, d + 2, h, w, case["cin"]), dtype=torch.bfloat16, device=DEV)
    g = torch.zeros((n, d + 2, h, w, case["cout"]), dtype=torch.bfloat16, device=DEV)
    x[:, 1:-1] = torch.randn((n, d, h, w, case["cin"]), generator=gen, device=DEV).clamp_min(0).bfloat16()
    live = torch.rand((n, d, h, w, case["cout"]), generator=gen, device=DEV) > 0.5
    g[:, 1:-1] = (torch.randn((n, d, h, w, case["cout"]), generator=gen, device=DEV) * live).bfloat16()
    wt = torch.randn((27, case["cout"], case["cin"]), generator=gen, device=DEV) * math.sqrt(2.0 / (27 * case["cin"]))
    bias = torch.randn(case["cout"], generator=gen, device=DEV) * 0.1
    return x, g, wt, bias


# ---------------------------------------------------------------------------------------------- states

class _Cabi:
    """A domain and a matrix through the C ABI, as a C++ or ctypes caller keeps them."""

    def __init__(self, ne):
        from esys_b200 import _lib as L
        self.L, self.lib = L, L.lib()
        d = len(ne)
        three = list(ne) + [1] * (3 - d)
        self.dom, self.mat = C.c_void_p(), C.c_void_p()
        L.set_stream_from_torch()
        L.check(self.lib.rg_domain_create(d, (C.c_int64 * 3)(*three), (C.c_double * 3)(0, 0, 0),
                                          (C.c_double * 3)(1, 1, 1), C.byref(self.dom)))
        n, nnz = C.c_int64(), C.c_int64()
        L.check(self.lib.rg_domain_info(self.dom, C.byref(n), C.byref(nnz), None, None, None))
        self.n, self.nnz = n.value, nnz.value
        L.check(self.lib.rg_matrix_create(self.dom, C.byref(self.mat)))
        self.rhs = torch.zeros(self.n, dtype=F64, device=DEV)
        self.x = torch.zeros(self.n, dtype=F64, device=DEV)

    def __del__(self):
        try:
            self.lib.rg_matrix_destroy(self.mat)
            self.lib.rg_domain_destroy(self.dom)
        except Exception:
            pass

    def assemble(self, coefs, kind, q):
        """coefs: name -> tensor; resets, assembles and constrains."""
        L, lib = self.L, self.lib
        L.set_stream_from_torch()
        L.check(lib.rg_matrix_reset(self.mat))
        self.rhs.zero_()
        c = [L.rg_coef(coefs[k].data_ptr(), kind) if k in coefs else L.rg_coef(None, L.RG_COEF_EMPTY) for k in "ABCDXY"]
        L.check(lib.rg_assemble_single(self.mat, C.c_void_p(self.rhs.data_ptr()), *[C.byref(v) for v in c]))
        L.check(lib.rg_insert_constraint(self.mat, C.c_void_p(self.rhs.data_ptr()), C.c_void_p(q.data_ptr()), None, 0))

    def solve(self, tol, layout):
        L, lib = self.L, self.lib
        o, d = L.rg_solver_opts(), L.rg_diag()
        lib.rg_solver_opts_default(C.byref(o))
        o.tolerance = tol
        o.mode, o.precision, o.layout = L.RG_MODE_STANDARD, L.RG_PREC_FP32_REFINE, layout
        L.check(lib.rg_solve(self.mat, C.c_void_p(self.rhs.data_ptr()), C.c_void_p(self.x.data_ptr()), C.byref(o),
                             C.byref(d)))
        return self.x

    def values(self):
        """The CSR values as a tensor on the matrix's own memory, which the tensor keeps alive."""
        p = C.c_void_p()
        self.L.check(self.lib.rg_matrix_values(self.mat, C.byref(p)))
        return torch.as_tensor(_View(self, p.value, self.nnz), device=DEV)


class _View:
    """Device doubles of `owner` for torch.as_tensor, whose tensor holds this object."""

    def __init__(self, owner, ptr, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(count),), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3, "stream": None}


def _domain(ne):
    from esys_b200 import ripley
    return ripley.Brick(*ne) if len(ne) == 3 else ripley.Rectangle(*ne)


def _on_function(dom, per_element, comps=()):
    """escript Data at the Gauss points from values per element."""
    from esys_b200 import escript
    q = 1 << dom.getDim()
    t = per_element.reshape(per_element.shape[0], 1, -1).expand(-1, q, -1).reshape(per_element.shape[0] * q, -1)
    return escript.Data._wrap(t.contiguous(), comps, escript.Function(dom))


def _prepare_pde(case, seed):
    from esys_b200 import escript
    inp = _pde_inputs(case, seed)
    dom = _domain(_ints(case["ne"]))
    d = dom.getDim()
    x = escript.Solution(dom).getX()
    values = {"A": _on_function(dom, inp["kappa"][:, None] * torch.eye(d, device=DEV, dtype=F64).reshape(1, -1), (d, d)),
              "Y": _on_function(dom, inp["y"]), "q": escript.whereZero(x[d - 1] - 1.0)}
    if case["terms"] == "robin":
        values["D"] = _on_function(dom, inp["d"])
        values["d"] = escript.Scalar(2.0, escript.FunctionOnBoundary(dom))
        values["y"] = escript.Scalar(inp["flux"], escript.FunctionOnBoundary(dom))
        values["r"] = escript.Scalar(inp["value"], escript.Solution(dom))
    pde = escript.LinearPDE(dom, numEquations=1, numSolutions=1)
    pde.getSolverOptions().setTolerance(case["tol"])
    return {"pde": pde, "values": values}


def _prepare_steps(case, seed):
    from esys_b200 import escript
    state = _prepare_pde(dict(case, terms="steps"), seed)
    pde, dom = state["pde"], state["pde"].getDomain()
    o = pde.getSolverOptions()
    o.setSolverMode(escript.SolverOptions.MODE_STANDARD)
    o.setMatrixLayout(escript.SolverOptions.LAYOUT_BAND)
    pde.setValue(D=_step_rate(_ints(case["ne"])), **state["values"])
    pde.getSystem()
    return {"pde": pde, "values": {"Y": state["values"]["Y"]}, "dom": dom}


def _step_rate(ne):
    """1/dt of an implicit step that spreads heat over some ten cells."""
    return float(max(ne)) ** 2 / 100.0


def _prepare_elastic(case, seed):
    from esys_b200 import escript
    mu, lam, load = _lame(case, seed)
    dom = _domain(_ints(case["ne"]))
    d = dom.getDim()
    a = _lame_tensor(mu, lam, d).permute(0, 4, 3, 2, 1).reshape(mu.numel(), -1)  # first index fastest
    x = escript.Solution(dom).getX()
    q = escript.Data(0.0, (d,), escript.Solution(dom), expanded=True)
    for i in range(d):
        q[i] = escript.whereZero(x[d - 1] - 1.0)
    pde = escript.LinearPDE(dom, numEquations=d, numSolutions=d)
    pde.getSolverOptions().setTolerance(case["tol"])
    return {"pde": pde, "values": {"A": _on_function(dom, a, (d,) * 4), "Y": _on_function(dom, load, (d,)), "q": q}}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pde":
        return dict(_prepare_pde(case, seed), case=case)
    if kind == "steps":
        return dict(_prepare_steps(case, seed), case=case)
    if kind == "elastic":
        return dict(_prepare_elastic(case, seed), case=case)
    if kind in ("refine", "aniso"):
        ne = _ints(case["ne"])
        s = _Cabi(ne)
        if kind == "refine":
            gen = _gen(seed)
            k = torch.exp(_field(ne, case["corr"], gen)).reshape(-1)
            a = k[:, None, None] * torch.eye(3, device=DEV, dtype=F64)
            coefs = {"A": a.contiguous(), "Y": _blobs(ne, gen).reshape(-1).contiguous()}
        else:
            a, dd, y = _aniso(case, seed)
            coefs = {"A": a.transpose(1, 2).contiguous(), "D": dd, "Y": y.contiguous()}
        return {"case": case, "sys": s, "coefs": coefs, "q": _top(ne)}
    if kind == "learned":
        from esys_b200 import warmstart as W
        ne = (case["edge"],) * 3
        gen = _gen(seed)
        prob = W.BrickProblem(case["edge"])
        return {"case": case, "prob": prob, "held": _Held([prob]), "start": W.WarmStart(W.UNet.load()),
                "kappa": torch.exp(_field(ne, case["corr"], gen)), "y": _blobs(ne, gen)}
    if kind == "batch":
        from esys_b200 import batch as B
        from esys_b200 import warmstart as W
        probs, rhs, keep = [], [], []
        for i, ne in enumerate(_batch_shapes(case)):
            gen = _gen(seed, i)
            p = W.BrickProblem(ne)
            k = torch.exp(_field(ne, 8.0, gen))
            b = torch.empty((case["nrhs"], p.n), dtype=F64, device=DEV)
            for r in range(case["nrhs"]):
                y = _blobs(ne, gen)
                p.assemble(k, y) if r == 0 else p.set_rhs(y)
                b[r].copy_(p.rhs)
            probs.append(p)
            rhs.append(b)
        solver = B.BatchSolver([p.mat for p in probs], case["nrhs"])
        solver.tune()
        return {"case": case, "probs": probs, "rhs": rhs, "x": [torch.zeros_like(b) for b in rhs], "solver": solver,
                "held": _Held([solver] + probs)}
    if kind == "assemble":
        return {"case": case, "sys": _Cabi(_ints(case["ne"])), "coefs": _assembly_inputs(case, seed),
                "q": _top(_ints(case["ne"]))}
    from esys_b200 import warmstart as W
    x, g, wt, bias = _conv_inputs(case, seed)
    wf, wd = wt.bfloat16(), torch.empty((27, case["cin"], case["cout"]), dtype=torch.bfloat16, device=DEV)
    W.weights_bf16(wt, wf, wd)
    return {"case": case, "W": W, "x": x, "g": g, "bias": bias, "wf": wf, "wd": wd, "y": torch.zeros_like(g),
            "dx": torch.zeros_like(x), "dw": torch.zeros_like(wt), "db": torch.zeros_like(bias),
            "partials": torch.zeros(1 << 24, dtype=torch.float32, device=DEV),
            "work": torch.zeros(592 * 128, dtype=torch.float32, device=DEV), "err": W.DeviceError(DEV)}


class _Held:
    """Closes what a state holds, in order."""

    def __init__(self, things):
        self.things = things

    def __del__(self):
        try:
            for t in self.things:
                t.close()
        except Exception:
            pass


# ---------------------------------------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("pde", "steps", "elastic"):
        state["pde"].setValue(**state["values"])
        return state["pde"].getSolution()._t
    if kind == "refine":
        s = state["sys"]
        s.assemble(state["coefs"], s.L.RG_COEF_PER_ELEMENT, state["q"])
        return s.solve(case["tol"], s.L.RG_LAYOUT_COEF)
    if kind == "aniso":
        s = state["sys"]
        s.assemble(state["coefs"], s.L.RG_COEF_PER_ELEMENT, state["q"])
        return s.solve(case["tol"], s.L.RG_LAYOUT_BAND)
    if kind == "learned":
        p = state["prob"]
        p.assemble(state["kappa"], state["y"])
        guess = state["start"].guess(state["kappa"].float(), state["y"].float(), p.shape, q=p.q)
        p.solve(tol=case["tol"], guess=guess, guess_sweeps=16)
        return p.x
    if kind == "batch":
        state["solver"].solve(state["rhs"], state["x"], tol=case["tol"])
        return state["x"]
    if kind == "assemble":
        s = state["sys"]
        s.assemble(state["coefs"], s.L.RG_COEF_EXPANDED if case["layout"] == "expanded" else s.L.RG_COEF_PER_ELEMENT,
                   state["q"])
        return [s.values(), s.rhs]
    W = state["W"]
    W.conv3(state["x"], state["wf"], state["bias"], state["y"], relu=True, err=state["err"])
    W.conv3_wgrad(state["x"], state["g"], state["dw"], state["partials"], err=state["err"])
    W.colsum(state["g"], None, state["db"], state["work"])
    W.conv3(state["g"], state["wd"], None, state["dx"], relu=False, mask=state["x"], err=state["err"])
    return [state["y"], state["dw"], state["db"], state["dx"]]


# ---------------------------------------------------------------------------------------------- work

def _iterations(ne, tol, rate=0.0):
    """Jacobi-PCG iterations to expect: proportional to the nodes per axis (fewer with a reaction term)."""
    m = sum(v + 1 for v in ne) / len(ne)
    full = 6.3 * m * math.log(tol) / math.log(1e-8) if len(ne) == 3 else 2.6 * m * math.log(tol) / math.log(1e-8)
    return min(full, 60.0) if rate else full


def work(case):
    """Inputs read once, outputs written once, and, for a solve, one read of the operator (one value per
    element and coefficient, or the stored rows where they are the operator) and of five vectors per
    iteration of Jacobi-PCG."""
    kind = case["kind"]
    if kind == "conv":
        w, h, d = _ints(case["grid"])
        p = case["n"] * w * h * d
        io = p * (2 * case["cin"] + 2 * case["cout"]) * 2 + 27 * case["cin"] * case["cout"] * 8
        return {"bytes": io, "flops": 3 * 2.0 * 27 * case["cin"] * case["cout"] * p}
    if kind == "batch":
        total = flops = 0.0
        for ne in _batch_shapes(case):
            n = math.prod(v + 1 for v in ne)
            it = _iterations(ne, case["tol"])
            total += n * (16.0 * case["nrhs"] + it * (4.0 + 20.0 * case["nrhs"]))
            flops += n * it * (54.0 + 10.0) * case["nrhs"]
        return {"bytes": total, "flops": flops}
    if kind == "learned":
        ne = (case["edge"],) * 3
    else:
        ne = _ints(case["ne"])
    d = len(ne)
    n, e, q = math.prod(v + 1 for v in ne), math.prod(ne), 1 << d
    rows = 3 ** d
    if kind == "assemble":
        comps = {"A": d * d, "B": d, "C": d, "D": 1, "X": d, "Y": 1}
        c = sum(comps[k] for k in case["coefs"])
        pts = q if case["layout"] == "expanded" else 1
        nnz = math.prod(3 * (v + 1) - 2 for v in ne)
        return {"bytes": 8.0 * (e * c * pts + nnz + 2 * n), "flops": 2.0 * e * q * q * q * d}
    if kind in ("refine", "learned"):
        it = _iterations(ne, case["tol"])
        return {"bytes": e * 80.0 + 16.0 * n + it * n * (4 + 20.0), "flops": it * n * 64.0}
    if kind == "aniso":
        it = _iterations(ne, case["tol"])
        return {"bytes": e * 88.0 + 16.0 * n + it * n * (4.0 * rows + 20.0), "flops": it * n * 64.0}
    if kind == "elastic":
        it = 1.5 * _iterations(ne, case["tol"])
        return {"bytes": 8.0 * e * q * (d ** 4 + d) + 8.0 * it * n * (rows * d * d + 5 * d),
                "flops": it * n * d * (2.0 * rows * d + 10)}
    it = _iterations(ne, case["tol"], 1.0 if kind == "steps" or case.get("terms") == "robin" else 0.0)
    coefs = 8.0 * e * q * (1 if kind == "steps" else d * d + 1)
    return {"bytes": coefs + 8.0 * it * n * (rows + 5), "flops": it * n * (2.0 * rows + 10)}


# ---------------------------------------------------------------------------------------------- 64 bits

def _q1(d, h):
    """Gauss points x nodes: shape functions N[q, k], gradients G[q, k, axis], the weight; bit a of q or k
    is the offset along axis a."""
    g = (0.5 - math.sqrt(3.0) / 6.0, 0.5 + math.sqrt(3.0) / 6.0)
    N = torch.zeros((1 << d, 1 << d), dtype=F64, device=DEV)
    G = torch.zeros((1 << d, 1 << d, d), dtype=F64, device=DEV)
    for q, k in itertools.product(range(1 << d), repeat=2):
        f = [(g[(q >> a) & 1] if (k >> a) & 1 else 1.0 - g[(q >> a) & 1]) for a in range(d)]
        N[q, k] = math.prod(f)
        for a in range(d):
            G[q, k, a] = (1.0 if (k >> a) & 1 else -1.0) / h[a] * math.prod(f[b] for b in range(d) if b != a)
    return N, G, math.prod(h) / (1 << d)


class _Bands:
    """A scalar operator on the node grid as 3^d bands (band by band over the nodes) and a right hand side."""

    def __init__(self, ne):
        self.ne, self.d = ne, len(ne)
        self.h = [1.0 / v for v in ne]
        self.nn = tuple(v + 1 for v in ne)
        self.shape = tuple(reversed(self.nn))
        self.n = math.prod(self.nn)
        self.band = torch.zeros((3 ** self.d,) + self.shape, dtype=F64, device=DEV)
        self.rhs = torch.zeros(self.shape, dtype=F64, device=DEV)

    def _at(self, k):
        """The nodes that are local node k of their element, as slices of a node array."""
        return tuple(slice((k >> a) & 1, self.ne[a] + ((k >> a) & 1)) for a in reversed(range(self.d)))

    def add(self, k, c, values):
        b = sum((1 + ((c >> a) & 1) - ((k >> a) & 1)) * 3 ** a for a in range(self.d))
        self.band[b][self._at(k)] += values.reshape(tuple(reversed(self.ne)))

    def isotropic(self, kappa):
        N, G, w = _q1(self.d, self.h)
        K = w * torch.einsum("qka,qca->kc", G, G)
        for k, c in itertools.product(range(1 << self.d), repeat=2):
            self.add(k, c, K[k, c] * kappa)

    def general(self, coefs, points):
        """coefs as in the C ABI, (elements, points, ...) or (elements, ...) without points."""
        N, G, w = _q1(self.d, self.h)
        v = {c: (t if points else t.unsqueeze(1).expand((t.shape[0], 1 << self.d) + t.shape[1:])) for c, t in coefs.items()}
        for k in range(1 << self.d):
            for c in range(1 << self.d):
                em = 0.0
                if "A" in v:
                    em = em + torch.einsum("eqji,qi,qj->e", v["A"], G[:, k], G[:, c])
                if "B" in v:
                    em = em + torch.einsum("eqi,qi,q->e", v["B"], G[:, k], N[:, c])
                if "C" in v:
                    em = em + torch.einsum("eqj,qj,q->e", v["C"], G[:, c], N[:, k])
                if "D" in v:
                    em = em + torch.einsum("eq,q->e", v["D"], N[:, k] * N[:, c])
                self.add(k, c, w * em)
            f = 0.0
            if "X" in v:
                f = f + torch.einsum("eqi,qi->e", v["X"], G[:, k])
            if "Y" in v:
                f = f + torch.einsum("eq,q->e", v["Y"], N[:, k])
            if "X" in v or "Y" in v:
                self.rhs[self._at(k)] += (w * f).reshape(tuple(reversed(self.ne)))

    def source(self, y):
        N, _, w = _q1(self.d, self.h)
        for k in range(1 << self.d):
            self.rhs[self._at(k)] += w * float(N[:, k].sum()) * y.reshape(tuple(reversed(self.ne)))

    def robin(self, dval, yval):
        """Face terms with constant d and y on all faces."""
        for ax in range(self.d):
            other = [a for a in range(self.d) if a != ax]
            N, _, w = _q1(len(other), [self.h[a] for a in other])
            M, F = w * torch.einsum("qk,qc->kc", N, N), w * N.sum(0)
            full = lambda m: sum(((m >> i) & 1) << a for i, a in enumerate(other))  # noqa: E731
            for side in (0, 1):
                for k in range(1 << len(other)):
                    at = list(self._at(full(k)))
                    pos = self.d - 1 - ax
                    at[pos] = slice(self.ne[ax] * side, self.ne[ax] * side + 1)
                    self.rhs[tuple(at)] += F[k] * yval
                    for c in range(1 << len(other)):
                        b = 3 ** ax + sum((1 + ((c >> i) & 1) - ((k >> i) & 1)) * 3 ** a for i, a in enumerate(other))
                        self.band[b][tuple(at)] += M[k, c] * dval

    def offsets(self):
        return [sum((o[a] - 1) * math.prod(self.nn[:a]) for a in range(self.d))
                for o in ([(b // 3 ** a) % 3 for a in range(self.d)] for b in range(3 ** self.d))]

    def mask(self):
        """Which bands have a neighbour, band by band over the nodes."""
        m = torch.ones((3 ** self.d,) + self.shape, dtype=torch.bool, device=DEV)
        for b in range(3 ** self.d):
            for a in range(self.d):
                o, ax = (b // 3 ** a) % 3, self.d - 1 - a
                if o != 1:
                    m[b].select(ax, 0 if o == 0 else self.nn[a] - 1).fill_(False)
        return m

    def constrain(self, q, r):
        """rhs -= A r on the fixed nodes, their rows and columns to those of the identity, rhs = r there."""
        q = q.reshape(-1) > 0
        band, rhs, off, mask = self.band.reshape(3 ** self.d, -1), self.rhs.reshape(-1), self.offsets(), self.mask()
        rows = torch.arange(self.n, device=DEV)
        for b, o in enumerate(off):
            ok = mask[b].reshape(-1)
            j = (rows + o).clamp(0, self.n - 1)
            fixed = ok & q[j]
            rhs -= torch.where(fixed, band[b] * r, torch.zeros_like(rhs))
            band[b][fixed | q] = 0.0
        band[3 ** self.d // 2][q] = 1.0
        rhs[q] = r

    def csr(self):
        off = torch.tensor(self.offsets(), device=DEV)
        m = self.mask().reshape(3 ** self.d, -1).t().contiguous()
        val = self.band.reshape(3 ** self.d, -1).t()[m]
        col = (torch.arange(self.n, device=DEV, dtype=torch.int32)[:, None] + off.int()[None, :])[m]
        ptr = torch.zeros(self.n + 1, dtype=torch.int32, device=DEV)
        ptr[1:] = m.sum(1).cumsum(0).int()
        return ptr, col, val

    def solve(self, rhs=None):
        """(n,) or, for right hand sides of shape (k, n), (k, n)."""
        b = (self.rhs.reshape(1, -1) if rhs is None else rhs).t().contiguous()
        diag = self.band[3 ** self.d // 2].reshape(-1, 1).clone()
        ptr, col, val = self.csr()
        self.band = None
        A = torch.sparse_csr_tensor(ptr, col, val, (self.n, self.n))
        x = _cg(A, b, 1.0 / diag)
        return x[:, 0] if rhs is None else x.t().contiguous()


def _cg(A, b, dinv, tol=2e-14, restarts=3, cap=12000):
    """Jacobi-PCG per column in 64 bits, restarted from the true residual."""
    mul = (lambda v: torch.mv(A, v[:, 0])[:, None]) if b.shape[1] == 1 else (lambda v: torch.sparse.mm(A, v))
    x = torch.zeros_like(b)
    goal = b.norm(dim=0) * tol
    for _ in range(restarts):
        r = b - mul(x)
        z = dinv * r
        p = z.clone()
        rho = (r * z).sum(0)
        for it in range(cap):
            s = mul(p)
            ps = (p * s).sum(0)
            alpha = torch.where(ps > 0, rho / ps, torch.zeros_like(rho))
            x += alpha * p
            r -= alpha * s
            z = dinv * r
            new = (r * z).sum(0)
            p = z + torch.where(rho > 0, new / rho, torch.zeros_like(rho)) * p
            rho = new
            if it % 32 == 31 and bool((r.norm(dim=0) <= goal).all()):
                break
    return x


def _exact_elastic(case, seed):
    ne = _ints(case["ne"])
    d = len(ne)
    mu, lam, load = _lame(case, seed)
    N, G, w = _q1(d, [1.0 / v for v in ne])
    nn = [v + 1 for v in ne]
    strides = [math.prod(nn[:a]) for a in range(d)]
    base = torch.zeros(tuple(reversed(ne)), dtype=torch.int64, device=DEV)
    for a in range(d):
        base = base + (torch.arange(ne[a], device=DEV) * strides[a]).reshape([-1 if t == d - 1 - a else 1 for t in range(d)])
    base = base.reshape(-1)
    node = torch.stack([base + sum(strides[a] * ((k >> a) & 1) for a in range(d)) for k in range(1 << d)], 1)
    n = math.prod(nn)
    A = _lame_tensor(mu, lam, d)
    em = w * torch.einsum("eijkl,qrj,qcl->erick", A, G, G)
    dof = (node[:, :, None] * d + torch.arange(d, device=DEV)).reshape(base.numel(), -1)
    m = dof.shape[1]
    rhs = torch.zeros(n * d, dtype=F64, device=DEV)
    rhs.index_add_(0, dof.reshape(-1), (w * torch.einsum("ei,k->eki", load, N.sum(0))).reshape(-1))
    fixed = (_top(ne) > 0).repeat_interleave(d)
    em = em.reshape(-1, m, m)
    free = (~fixed[dof]).to(F64)
    em = em * free[:, :, None] * free[:, None, :]
    rows, cols = dof[:, :, None].expand(-1, m, m).reshape(-1), dof[:, None, :].expand(-1, m, m).reshape(-1)
    every = torch.nonzero(fixed)[:, 0]
    ind = torch.stack([torch.cat([rows, every]), torch.cat([cols, every])])
    val = torch.cat([em.reshape(-1), torch.ones(every.numel(), dtype=F64, device=DEV)])
    S = torch.sparse_coo_tensor(ind, val, (n * d, n * d)).coalesce()
    at = S.indices()
    diag = torch.zeros(n * d, dtype=F64, device=DEV)
    on = at[0] == at[1]
    diag[at[0][on]] = S.values()[on]
    rhs[fixed] = 0.0
    return _cg(S.to_sparse_csr(), rhs[:, None], 1.0 / diag[:, None])[:, 0].reshape(n, d)


def _exact_conv(case, seed):
    x, g, wt, bias = _conv_inputs(case, seed)
    wd = wt.bfloat16().double()
    xi, gi = x[:, 1:-1], g[:, 1:-1]
    n, d, h, w, _ = xi.shape

    def shifted(t, kd, kh, kw):
        """t(p + (kd, kh, kw)), zero outside."""
        return torch.nn.functional.pad(t.double(), (0, 0, 1, 1, 1, 1, 1, 1))[:, 1 + kd:1 + kd + d, 1 + kh:1 + kh + h,
                                                                            1 + kw:1 + kw + w]

    y = bias.double().expand(n, d, h, w, -1).clone()
    dx = torch.zeros(xi.shape, dtype=F64, device=DEV)
    dw = torch.empty(wt.shape, dtype=F64, device=DEV)
    for tap, (kd, kh, kw) in enumerate(itertools.product((-1, 0, 1), repeat=3)):
        xs = shifted(xi, kd, kh, kw)
        y += xs @ wd[tap].t()
        dw[tap] = gi.double().reshape(-1, gi.shape[-1]).t() @ xs.reshape(-1, xs.shape[-1])
        dx += shifted(gi, -kd, -kh, -kw) @ wd[tap]
    out_y, out_dx = torch.zeros(g.shape, dtype=F64, device=DEV), torch.zeros(x.shape, dtype=F64, device=DEV)
    out_y[:, 1:-1] = y.clamp_min(0)
    out_dx[:, 1:-1] = torch.where(xi > 0, dx, torch.zeros_like(dx))
    return [out_y, dw, gi.double().sum((0, 1, 2, 3)), out_dx]


def exact(case, seed):
    kind = case["kind"]
    if kind == "conv":
        return _exact_conv(case, seed)
    if kind == "elastic":
        return _exact_elastic(case, seed)
    if kind == "batch":
        out = []
        for i, ne in enumerate(_batch_shapes(case)):
            gen = _gen(seed, i)
            b = _Bands(ne)
            b.isotropic(torch.exp(_field(ne, 8.0, gen)))
            rhs = torch.empty((case["nrhs"], b.n), dtype=F64, device=DEV)
            q = _top(ne)
            for r in range(case["nrhs"]):
                b.rhs.zero_()
                b.source(_blobs(ne, gen))
                rhs[r] = b.rhs.reshape(-1)
            b.constrain(q, 0.0)
            rhs[:, q > 0] = 0.0
            out.append(b.solve(rhs))
        return out
    ne = (case["edge"],) * 3 if kind == "learned" else _ints(case["ne"])
    b = _Bands(ne)
    if kind == "assemble":
        b.general(_assembly_inputs(case, seed), case["layout"] == "expanded")
        b.constrain(_top(ne), 0.0)
        return [b.csr()[2], b.rhs.reshape(-1)]
    value = 0.0
    if kind == "aniso":
        a, dd, y = _aniso(case, seed)
        b.general({"A": a.transpose(1, 2), "D": dd, "Y": y}, False)
    elif kind in ("refine", "learned"):
        gen = _gen(seed)
        b.isotropic(torch.exp(_field(ne, case["corr"], gen)))
        b.source(_blobs(ne, gen))
    else:
        inp = _pde_inputs(case, seed)
        b.isotropic(inp["kappa"])
        b.source(inp["y"])
        if kind == "steps":
            b.general({"D": torch.full_like(inp["kappa"], _step_rate(ne))}, False)
        elif case["terms"] == "robin":
            b.general({"D": inp["d"]}, False)
            b.robin(2.0, inp["flux"])
            value = inp["value"]
    b.constrain(_top(ne), value)
    x = b.solve()
    return x if kind in ("refine", "aniso", "learned") else x[:, None]
