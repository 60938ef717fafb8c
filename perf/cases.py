"""Performance cases of the per-cell chemistry solve.

Each case is one call (or one batch of serving requests) as a host model makes it: a
mechanism, a number of grid cells, a host time step, the precision and the entry point.
``listed`` gives the fixed cases, ``draw`` more of the same ranges; ``prepare`` builds the
solver and its inputs, ``run`` makes the call once, ``work`` counts what a call cannot do
without and ``exact`` integrates the same cells in 64 bits with plain torch.

Keys of a case:

* ``mech``: one of ``MECHS`` (the packed mechanisms of ``tests/golden`` and the synthetic
  200-species mechanism), or ``mix`` for the serving mix of two mechanisms;
* ``cells``: cells of the call (columns of a serving batch have 10-200 cells each);
* ``inputs``: ``physical`` (around the cb05 test's initial concentrations, a factor of three
  either way) or ``log_uniform`` (every species log-uniform over 1e-6..1e2 ppm, the
  benchmark's cells, a quarter of which run into the step limit);
* ``dt``: the host step in seconds;
* ``mixed``: FP32 Jacobian and LU beside an FP64 state, or FP64 throughout;
* ``max_steps``: internal steps after which a cell is given up (the library's default is 10000);
* ``entry``: ``host`` (``solver_run`` on host arrays), ``device`` (device-resident arrays,
  one graph launch, longest cells first, as the benchmark runs it) or ``server``.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from camp_b200.cells import make_cells
from camp_b200.mechanism import Mechanism
from camp_b200.serve import Server
from camp_b200.solver import FP64, MIXED, Solver
from camp_b200.synth import load_synthetic

GOLDEN = os.path.join("tests", "golden")
MECHS = ("cb05cl_ae5", "monarch_mod37_gas", "monarch_mod37_soa", "monarch_mod37_aero",
         "monarch_mod37_shipped", "synthetic")
RTOL, ATOL = 1.0e-4, 1.0e-8
SPREAD = 3.0  # physical cells: factor either way around the initial concentrations
TRACE = 1.0e-6  # ppm of a gas species that the cb05 test's initial state does not have

_mechs: dict[str, tuple] = {}


def _mech(name: str):
    """(mechanism, photolysis base rates or None)."""
    if name not in _mechs:
        if name == "synthetic":
            with tempfile.TemporaryDirectory() as d:
                _mechs[name] = load_synthetic(d, 200, 600)
        else:
            _mechs[name] = (Mechanism.load(os.path.join(GOLDEN, name + ".mech.json")), None)
    return _mechs[name]


def listed():
    def case(name, mech, cells, dt, mixed, entry, inputs="physical", max_steps=10000):
        return {"name": name, "mech": mech, "cells": cells, "inputs": inputs, "dt": dt,
                "mixed": mixed, "max_steps": max_steps, "entry": entry}

    cb05, gas, soa, aero, shipped = MECHS[:5]
    return [
        # a box model: the smallest call there is, latency alone
        case("box", cb05, 1, 60.0, False, "host"),
        # one column of a regional model through the drop-in entry point
        case("column", cb05, 73, 300.0, True, "host"),
        # a host rank's tile of columns
        case("tile", cb05, 2001, 300.0, False, "host"),
        # a whole domain kept on the device, in both precisions; the mixed one has the
        # benchmark's number of cells
        case("domain", cb05, 20000, 60.0, False, "device"),
        case("domain_mixed", cb05, 100000, 60.0, True, "device"),
        # the benchmark's own inputs: hard cells beside easy ones, a long tail
        case("benchmark", cb05, 1024, 60.0, True, "device", "log_uniform"),
        # MONARCH's mechanism with deposition and emission, then with its aerosol parts
        case("mod37_gas", gas, 5000, 300.0, True, "device"),
        case("mod37_soa", soa, 1500, 300.0, False, "host"),
        case("mod37_aero", aero, 1000, 60.0, True, "device"),
        # the shipped test configuration with its sub-models, for which FP64 is the form to use;
        # a few of its cells never finish, and a host gives those up
        case("mod37_shipped", shipped, 500, 60.0, False, "host", max_steps=4000),
        # a large mechanism, whose LU needs a thread block per cell
        case("synthetic", "synthetic", 592, 0.5, True, "device"),
        # columns of two mechanisms arriving together at the serving loop
        case("serving", "mix", 800, 300.0, True, "server"),
    ]


# the most cells of a drawn case, by mechanism (and of the benchmark's hard inputs)
_MOST = {"cb05cl_ae5": 60000, "monarch_mod37_gas": 20000, "monarch_mod37_soa": 4000,
         "monarch_mod37_aero": 3000, "monarch_mod37_shipped": 1200, "synthetic": 1000,
         "mix": 2000}
_MOST_HARD = 1500


def draw(rng):
    mech = rng.choice(("cb05cl_ae5", "cb05cl_ae5") + MECHS + ("mix",))
    inputs = "log_uniform" if mech == "cb05cl_ae5" and rng.random() < 0.2 else "physical"
    most = _MOST_HARD if inputs == "log_uniform" else _MOST[mech]
    least = 20 if mech == "mix" else 1
    cells = int(round(math.exp(rng.uniform(math.log(least), math.log(most)))))
    if mech == "synthetic":
        dt = rng.choice((0.25, 0.5))
    elif inputs == "log_uniform" or "aero" in mech or "shipped" in mech:
        dt = rng.choice((30.0, 60.0))
    else:
        dt = rng.choice((60.0, 120.0, 300.0, 900.0) if cells <= 10000 else (60.0, 120.0))
    mixed = rng.random() < 0.5 and mech != "monarch_mod37_shipped"
    max_steps = rng.choice((2000, 4000)) if "shipped" in mech else 10000
    entry = "server" if mech == "mix" else rng.choice(("host", "device"))
    return {"mech": mech, "cells": cells, "inputs": inputs, "dt": dt, "mixed": mixed,
            "max_steps": max_steps, "entry": entry}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _cells(name: str, n: int, inputs: str, seed: int):
    mech, base = _mech(name)
    if name == "synthetic":
        return make_cells(mech, n, seed, conc_lo=1.0e-8, photo_base=base)
    cells = make_cells(mech, n, seed)
    if inputs == "physical":
        # gas species at the cb05 test's initial state; aerosol species keep make_cells' loading
        init = {s: p["init conc"] for s, p in _mech("cb05cl_ae5")[0].species_props.items()
                if "init conc" in p}
        rng = np.random.Generator(np.random.PCG64(seed + 0x5EED))
        fac = np.exp(rng.uniform(-math.log(SPREAD), math.log(SPREAD), cells.state.shape))
        for i, s in enumerate(mech.species):
            if "." in s or mech.var_type[i] not in (1, 2):
                continue  # a species of an aerosol phase
            if mech.var_type[i] == 2 or s in ("M", "N2", "O2", "H2", "CH4"):
                cells.state[:, i] = init.get(s, 0.0)
            else:
                cells.state[:, i] = init.get(s, TRACE) * fac[:, i]
    return cells


def _solver(name: str, n: int, case: dict) -> Solver:
    mech, _ = _mech(name)
    s = Solver(mech, n)
    s.initialize(abs_tol=np.full(mech.n_state_var, ATOL), rel_tol=RTOL,
                 max_steps=case["max_steps"])
    s.set_precision(MIXED if case["mixed"] else FP64)
    return s


def _columns(case: dict):
    """(mechanism, cells) of a serving batch: columns of 10-200 cells, every third one of the
    mechanism with aerosol."""
    left, out, size = case["cells"], [], (72, 19, 200, 47, 101, 10, 133)
    while left > 0:
        n = min(left, size[len(out) % len(size)])
        out.append(("monarch_mod37_soa" if len(out) % 3 == 2 else "cb05cl_ae5", n))
        left -= n
    return out


def prepare(case, seed):
    n, st = case["cells"], dict(case)
    if case["entry"] == "server":
        st["server"] = Server(n_slots=4, device_mb=1024.0, host_mb=256.0)
        st["solvers"] = {m: _solver(m, 1, case)
                         for m in ("cb05cl_ae5", "monarch_mod37_soa")}
        st["index"] = {m: st["server"].add_solver(s) for m, s in st["solvers"].items()}
        st["columns"] = [(m, _cells(m, k, "physical", seed * 64 + i))
                         for i, (m, k) in enumerate(_columns(case))]
        return st
    cells = _cells(case["mech"], n, case["inputs"], seed)
    s = st["solver"] = _solver(case["mech"], n, case)
    if case["entry"] == "device":
        st["state"] = torch.from_numpy(cells.state).cuda()
        st["env"] = torch.from_numpy(cells.env).cuda()
        s.set_photo_rates_device(torch.from_numpy(
            np.ascontiguousarray(cells.photo_rates)).cuda(), n)
        s.set_graph(True)
        s.set_cost_ordering(True)
        st["stream"] = torch.cuda.Stream()
    else:
        st["state"], st["env"] = cells.state, cells.env
        s.set_photo_rates(cells.photo_rates)
    return st


def run(st):
    if st["entry"] == "server":
        srv = st["server"]
        ids = [srv.submit(st["index"][m], c.state.copy(), c.env, c.photo_rates, 0.0, st["dt"])
               for m, c in st["columns"]]
        return [srv.wait(i)[2] for i in ids]
    s = st["solver"]
    if st["entry"] == "device":
        with torch.cuda.stream(st["stream"]):
            y = st["state"].clone()
            status = s.run_device(y, st["env"], st["cells"], 0.0, st["dt"], st["stream"])
    else:
        y = st["state"].copy()
        status = s.solve(y, st["env"], 0.0, st["dt"])
    return {"state": y, "status": status}


# ---------------------------------------------------------------------------
# Compulsory work
# ---------------------------------------------------------------------------
# internal steps that a cell takes on average, from runs of these cases
_STEPS = {"log_uniform": 3000, "physical": 70, "synthetic": 470, "monarch_mod37_shipped": 600}


def work(case):
    """Bytes: state, environment and host-set rates read once, dependent species written
    once.  Operations: per internal step one evaluation of every rate and of every
    participant's sum, and one pair of triangular solves over the solver Jacobian's entries."""
    parts = _columns(case) if case["entry"] == "server" else [(case["mech"], case["cells"])]
    nbytes = flops = 0
    for name, n in parts:
        mech, _ = _mech(name)
        dep = int(np.count_nonzero(mech.var_type == 1))
        nbytes += n * 8 * (mech.n_state_var + 2 + len(mech.rate_columns()) + dep)
        terms = sum(int(r.ints[0]) + int(r.ints[1]) if r.rxn_type <= 5 else 2 for r in mech.rxns)
        steps = _STEPS.get(name, _STEPS[case["inputs"]])
        flops += n * steps * (4 * terms + 2 * 10 * dep)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# 64-bit solution: mass-action kinetics by extrapolated linearly implicit Euler
# ---------------------------------------------------------------------------
_EXACT = {"cb05cl_ae5": 100, "synthetic": 8}  # most cells
_ORDERS = (1, 2, 3, 4, 5, 6, 7, 8)  # substeps of the extrapolation table's rows


def _rate(r, T, P, base):
    """Rate constants of one reaction over the cells (T K, P Pa)."""
    f = [float(v) for v in r.floats]
    nr = int(r.ints[0])

    def law(a, b, c):
        return a * torch.exp(c / T) * (T / 300.0) ** b

    if r.rxn_type == 1:  # Arrhenius
        return (f[0] * torch.exp(f[2] / T) * (T / f[3]) ** f[1] * (1.0 + f[4] * P)
                * (f[5] * P / T) ** (nr - 1))
    if r.rxn_type == 2:  # Troe
        conv = f[9] * P / T
        k0 = law(f[0], f[1], f[2]) * conv
        ratio = k0 / law(f[3], f[4], f[5])
        return (k0 / (1.0 + ratio) * f[6] ** (1.0 / (1.0 + (torch.log10(ratio) / f[7]) ** 2))
                * conv ** (nr - 1) * f[8])
    if r.rxn_type == 3:  # CMAQ H2O2
        conv = f[6] * P / T
        return (law(*f[0:3]) + law(*f[3:6]) * conv) * conv ** (nr - 1)
    if r.rxn_type == 4:  # CMAQ OH + HNO3
        conv = f[10] * P / T
        k2, k3 = law(*f[3:6]), law(*f[6:9]) * conv
        return (law(*f[0:3]) + k3 / (1.0 + k3 / k2)) * conv ** (nr - 1) * f[9]
    return f[0] * base  # photolysis


_YIELDS = {1: 6, 2: 10, 3: 7, 4: 11, 5: 1}  # first yield in a reaction's floats


def exact(case, seed):
    name = case["mech"]
    if case["cells"] > _EXACT.get(name, 0) or case["inputs"] != "physical":
        return None  # too long, or (hard inputs) a solution that the step size decides
    mech, _ = _mech(name)
    cells = _cells(name, case["cells"], case["inputs"], seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")

    def on(a):
        return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)

    T, P, photo = on(cells.env[:, 0]), on(cells.env[:, 1]), on(cells.photo_rates)
    ns, nrx = mech.n_state_var, len(mech.rxns)
    column = {rxn: j for j, (_, rxn, *_) in enumerate(mech.rate_columns())}
    k = torch.empty((len(T), nrx), dtype=torch.float64, device=dev)
    # reactants as columns of the state extended by a column of ones, and net yields
    react = torch.full((nrx, 3), ns, dtype=torch.int64)
    net = torch.zeros((nrx, ns), dtype=torch.float64)
    var = torch.as_tensor(mech.var_type == 1)
    for i, r in enumerate(mech.rxns):
        k[:, i] = _rate(r, T, P, photo[:, column[i]] if i in column else None)
        nr, npr = int(r.ints[0]), int(r.ints[1])
        at = 3 if r.rxn_type == 5 else 2
        for j in range(nr):
            s = int(r.ints[at + j]) - 1
            react[i, j] = s
            net[i, s] -= 1.0
        for j in range(npr):
            net[i, int(r.ints[at + nr + j]) - 1] += float(r.floats[_YIELDS[r.rxn_type] + j])
    net = (net * var).to(dev)
    react = react.to(dev)
    rows = torch.arange(nrx, device=dev)
    eye = torch.eye(ns, dtype=torch.float64, device=dev)
    one = torch.ones((len(T), 1), dtype=torch.float64, device=dev)

    def f(y):
        return (k * torch.cat((y, one), 1)[:, react].prod(2)) @ net

    def jac(y):
        x = torch.cat((y, one), 1)[:, react]
        d = torch.zeros((len(y), nrx, ns + 1), dtype=torch.float64, device=dev)
        for j in range(3):
            a, b = [m for m in range(3) if m != j]
            d[:, rows, react[:, j]] += k * x[:, :, a] * x[:, :, b]
        return net.T @ d[:, :, :ns]

    y = on(cells.state).clamp(min=1.0e-30)
    t = torch.zeros_like(T)
    h = torch.full_like(T, 1.0e-9)
    end = case["dt"]
    for _ in range(4000):
        left = end - t
        if not bool((left > 0.0).any()):
            break
        h = torch.minimum(h, left)
        J = jac(y)
        row = []
        for j, m in enumerate(_ORDERS):
            step = h / m
            lu, piv = torch.linalg.lu_factor(eye - step[:, None, None] * J)
            u = y
            for _ in range(m):
                u = u + torch.linalg.lu_solve(lu, piv, (step[:, None] * f(u))[..., None])[..., 0]
            new = [u]
            for q in range(1, j + 1):
                new.append(new[-1] + (new[-1] - row[q - 1]) / (m / _ORDERS[j - q] - 1.0))
            row = new
        err = ((row[-1] - row[-2]).abs() / (1.0e-9 * y.abs() + 1.0e-15)).amax(1)
        err = torch.nan_to_num(err, nan=1.0e30, posinf=1.0e30).clamp(min=1.0e-12)
        ok = (err <= 1.0) & (h > 0.0)
        y = torch.where(ok[:, None], row[-1], y)
        t = torch.where(ok, torch.where(h >= left, torch.full_like(t, end), t + h), t)
        h = torch.where(left > 0.0, h * (0.8 * err ** (-1.0 / len(_ORDERS))).clamp(0.1, 4.0), h)
    if bool((t < end).any()):
        return None
    out = y.clamp(min=0.0)
    return {"state": out if case["entry"] == "device" else out.cpu().numpy(), "status": None}
