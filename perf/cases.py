"""The work whose speed this repository watches: the calls a program makes on the GPU path.

An electromagnetics program holds a pencil (A, B) of a cavity (edge elements on a Yee grid or on
tetrahedra, filled with a dielectric that varies in space) and
  * sweeps a shift: factorizes A - sigma B and solves a block of sources        ("sweep")
  * solves block after block on the factors that it keeps                       ("solve")
  * asks how many modes lie below a frequency                                   ("count")
  * checks its solutions by the residual of the shifted operator                ("residual")
  * asks for certified modes through a session that keeps the pencil            ("modes").
Sizes run from a few hundred unknowns (a unit test, a coarse cell) over the named boxes of
hsolve_b200.gen to about 3e5 unknowns; block widths from one source to 16. The sparsity pattern of
a case is fixed, everything else (dielectric, shift, sources) comes from the seed.
"""
import functools
import math

import numpy as np
import torch

import hsolve_b200
from hsolve_b200 import _native
from hsolve_b200.gen import nedelec, yee

LENGTHS = {"box": (1.0, 0.75, 0.55), "cube": (1.0, 1.0, 1.0), "tet": (2.0, 1.0, 0.5)}
SMALLEST, LARGEST = 700, 220_000  # unknowns of a drawn case


def _case(name, op, mesh, cells, form, p, **more):
    return {"name": name, "op": op, "mesh": mesh, "nx": cells[0], "ny": cells[1], "nz": cells[2], "form": form, "p": p,
            **more}


def listed():
    return [
        # the check of one solved block on the 20^3 cavity: one short kernel, launch and wait
        _case("residual_cube20_p8", "residual", "cube", (20, 20, 20), "standard", 8),
        # mode counts: a coarse cell, and an end of the headline interval
        _case("count_737", "count", "box", (8, 7, 6), "generalized", 0),
        _case("count_box1e5", "count", "box", (44, 34, 26), "generalized", 0),
        # one point of a frequency sweep, from the meshes of the tests to the largest
        _case("sweep_3021_p4", "sweep", "box", (14, 11, 8), "generalized", 4),
        _case("sweep_cube20_p8", "sweep", "cube", (20, 20, 20), "standard", 8),
        _case("sweep_box1e5_p8", "sweep", "box", (44, 34, 26), "generalized", 8),
        _case("sweep_box3e5_p8", "sweep", "box", (60, 47, 36), "generalized", 8),
        # further sources on held factors: one source, the Krylov block, the widest block on tetrahedra
        _case("solve_box1e4_p1", "solve", "box", (20, 16, 12), "generalized", 1),
        _case("solve_box1e5_p8", "solve", "box", (44, 34, 26), "generalized", 8),
        _case("solve_tet1e5_p16", "solve", "tet", (50, 25, 13), "generalized", 16),
        # certified modes: FP32 operator factors with FP64 refinement, and the headline interval
        _case("modes_box1e4_single", "modes", "box", (20, 16, 12), "generalized", 4, target="nearest",
              precision="single"),
        _case("modes_box1e5", "modes", "box", (44, 34, 26), "generalized", 4, target="interval", precision="double"),
    ]


def draw(rng):
    op = rng.choice(["sweep", "sweep", "sweep", "solve", "solve", "count", "count", "residual", "modes"])
    most = 30_000 if op == "modes" else LARGEST
    n = math.exp(rng.uniform(math.log(SMALLEST), math.log(most)))
    mesh = rng.choice(["box", "box", "cube", "tet"]) if op != "modes" else "box"
    form = "standard" if mesh == "cube" or (mesh == "box" and rng.random() < 0.3) else "generalized"
    # cells of the wanted number of unknowns, at ratios around those of the named boxes
    ratio = [1.0, rng.uniform(0.6, 1.0), rng.uniform(0.4, 0.9)] if mesh != "cube" else [1.0, 1.0, 1.0]
    per_cell = 3.0 if mesh != "tet" else 6.2
    c = (n / per_cell / math.prod(ratio)) ** (1.0 / 3.0)
    cells = [max(5 if mesh != "tet" else 3, round(c * r)) for r in ratio]
    if op == "modes":
        target, precision = rng.choice([("interval", "double"), ("nearest", "double"), ("nearest", "single")])
        case = _case("", op, mesh, cells, "generalized", 4, target=target, precision=precision)
    else:
        case = _case("", op, mesh, cells, form, 0 if op == "count" else rng.randint(1, 16))
    del case["name"]
    return case


# ------------------------------------------------------------------------------------ inputs

def _cells(case):
    return case["nx"], case["ny"], case["nz"]


@functools.lru_cache(maxsize=3)
def _vacuum(mesh, cells):
    """The empty cavity's (A, B) and the relative place of every edge, kept between seeds."""
    if mesh == "tet":
        a, b = nedelec.pencil(nedelec.TetBox(cells, LENGTHS[mesh]))
        at = np.stack([np.linspace(0.0, 1.0, a.shape[0])] * 3, axis=1)
        return a.tocsr(), b.tocsr(), at
    a, b = yee.assemble(yee.Box(cells, LENGTHS[mesh]))
    at = []
    for d in range(3):  # the middles of the edges along d, in the generator's order
        axes = [(np.arange(c) + 0.5) / c if q == d else np.arange(1, c) / c for q, c in enumerate(cells)]
        at.append(np.stack([g.ravel() for g in np.meshgrid(*axes, indexing="ij")], axis=1))
    return a.tocsr(), b.tocsr(), np.concatenate(at)


def _scaled(m, s):
    """diag(s) m diag(s)."""
    out = m.copy()
    out.data = m.data * np.repeat(s, np.diff(m.indptr)) * s[m.indices]
    return out


def _pencil(case, rng):
    """A and B (None in the standard form) of the cavity with this seed's filling: three smooth
    bodies of up to twice the permittivity, or for the interval target an even one (its spectrum
    is known in closed form, and the interval is the empty cavity's [40, 200] for it)."""
    a, b, at = _vacuum(case["mesh"], _cells(case))
    eps = np.full(a.shape[0], 1.0 + 0.05 * rng.random())
    if case.get("target") != "interval":
        for _ in range(3):
            where, width = rng.uniform(0.2, 0.8, 3), rng.uniform(0.1, 0.3)
            eps += rng.uniform(0.2, 1.0) * np.exp(-np.sum((at - where) ** 2, axis=1) / (2 * width**2))
    if case["form"] == "standard":
        return _scaled(a, 1.0 / np.sqrt(b.diagonal() * eps)), None, eps[0]
    return a, _scaled(b, np.sqrt(eps)), eps[0]


def _shift(rng):
    return float(rng.uniform(60.0, 180.0))


def _times(a, b, sigma, x):
    return a @ x - sigma * (x if b is None else b @ x)


def _block(v):
    """n x p on the host to the GPU, column after column."""
    return torch.from_numpy(np.ascontiguousarray(v.T)).cuda()


def _host(case, seed):
    """What the seed decides, on the host: the pencil, the shift, the fields and the filling."""
    rng = np.random.default_rng(seed)
    a, b, eps = _pencil(case, rng)
    sigma = _shift(rng)
    fields = rng.standard_normal((a.shape[0], max(1, case["p"])))
    return a, b, sigma, fields, eps, rng


def prepare(case, seed):
    a, b, sigma, fields, eps, rng = _host(case, seed)
    op, n, p = case["op"], a.shape[0], case["p"]
    if op == "residual":
        y = rng.standard_normal(fields.shape)
        return {"op": op, "a": _native.DeviceCsr(a), "b": None if b is None else _native.DeviceCsr(b), "sigma": sigma,
                "x": _block(fields), "y": _block(y), "r": torch.empty(p, n, dtype=torch.float64, device="cuda"),
                "omega": torch.empty(p, dtype=torch.float64, device="cuda")}
    if op == "modes":
        return {"op": op, "session": hsolve_b200.Session(a, b), "sources": fields if b is None else b @ fields,
                "target": {"lower": 40.0 / eps, "upper": 200.0 / eps} if case["target"] == "interval" else
                {"sigma": sigma, "k": 10},
                "config": {"factor_precision": case["precision"]}}
    f = hsolve_b200.Factorization(device=0)
    f.analyze(a, b, 1.0, -sigma)
    state = {"op": op, "f": f, "sigma": sigma, "n": n, "p": p}
    if op != "count":
        state["rhs"] = _block(_times(a, b, sigma, fields))
        state["x"] = torch.empty_like(state["rhs"])
    if op == "solve":
        f.factorize(1.0, -sigma)
    return state


def run(state):
    op = state["op"]
    if op == "residual":
        _native.shifted_residual_device(state["a"], state["b"], state["sigma"], state["x"], state["y"], state["r"],
                                        state["omega"])
        return {"r": state["r"], "omega": state["omega"]}
    if op == "modes":
        # A multiple mode's vectors are any basis of their space, so what is returned is what a
        # program does with them: the expansion of its sources in the modes.
        got = state["session"].solve(**state["target"], config=state["config"])
        v = got.eigenvectors
        return {"eigenvalues": got.eigenvalues, "expansion": v @ (v.T @ state["sources"]),
                "certified": int(got.success)}
    f = state["f"]
    if op == "count":
        c = f.count(1.0, -state["sigma"])
        return {"inertia": [c.neg, c.zero, c.pos]}
    out = {}
    if op == "sweep":
        f.factorize(1.0, -state["sigma"])
        c = f.inertia()
        out["inertia"] = [c.neg, c.zero, c.pos]
    state["x"].copy_(state["rhs"])
    f.solve_device(state["x"].data_ptr(), state["p"], state["n"])
    out["x"] = state["x"]
    return out


# ------------------------------------------------------------------- what a pass cannot do without

@functools.lru_cache(maxsize=16)
def _analysis(mesh, cells, form):
    a, b, _ = _vacuum(mesh, cells)
    m = a if form == "standard" else abs(a) + abs(b)
    return a.shape[0], a.nnz, b.nnz, _native.symbolic_stats(m)


def work(case):
    n, nnz_a, nnz_b, s = _analysis(case["mesh"], _cells(case), case["form"])
    p, single = case["p"], case.get("precision") == "single"
    pencil = 12.0 * (nnz_a + (nnz_b if case["form"] == "generalized" else 0))
    factor = 8.0 * s["nnz_l"]
    one_solve = 2 * factor + 2 * 8.0 * n * p  # the factors forward and backward, the block in and out
    if case["op"] == "residual":
        return {"bytes": pencil + 3 * 8.0 * n * p, "flops": 8.0 * nnz_a * p}
    if case["op"] == "count":
        return {"bytes": pencil, "flops": s["flops"]}
    if case["op"] == "solve":
        return {"bytes": one_solve, "flops": 4.0 * s["nnz_l"] * p}
    if case["op"] == "sweep":
        return {"bytes": pencil + factor + one_solve, "flops": s["flops"] + 4.0 * s["nnz_l"] * p}
    # two counts and a factorization; 25 blocks of eight through the factors, or 10 of a small target
    blocks = 25 if case["target"] == "interval" else 10
    return {"bytes": pencil + factor * (0.5 if single else 1.0) * (1 + 2 * blocks),
            "flops": 3 * s["flops"] + 32.0 * s["nnz_l"] * blocks}


# --------------------------------------------------------------------------- the same in 64 bits

def _spectrum(cells, lengths):
    """Closed form of the empty box: (2 / h sin(m pi / 2N))^2 summed over the axes, two
    modes where all m are positive, one where one of them is zero."""
    t = [(2.0 * c / size * np.sin(np.arange(c) * np.pi / (2 * c))) ** 2 for c, size in zip(cells, lengths)]
    total = t[0][:, None, None] + t[1][None, :, None] + t[2][None, None, :]
    m = [np.arange(c) > 0 for c in cells]
    some = m[0][:, None, None].astype(int) + m[1][None, :, None] + m[2][None, None, :]
    return np.sort(np.concatenate([np.repeat(total[some == 3], 2), total[some == 2]]))


def exact(case, seed):
    a, b, sigma, fields, eps, rng = _host(case, seed)
    if case["op"] == "count":
        return None
    if case["op"] == "residual":
        y = rng.standard_normal(fields.shape)
        s = fields + sigma * y
        r = (s if b is None else b @ s) - a @ y
        size = (abs(s) if b is None else abs(b) @ abs(s)) + abs(a) @ abs(y)
        return {"r": np.ascontiguousarray(r.T), "omega": np.max(np.abs(r) / size, axis=0)}
    if case["op"] == "modes":
        if case["target"] != "interval":
            return None
        w = _spectrum(_cells(case), LENGTHS[case["mesh"]])
        return {"eigenvalues": w[(w >= 40.0) & (w <= 200.0)] / eps, "expansion": None, "certified": 1}
    x = np.ascontiguousarray(fields.T)  # the sources were made from these fields
    return {"x": x} if case["op"] == "solve" else {"inertia": [None, None, None], "x": x}
