"""The warp kernel's round-structured gathers, factorization and solves at the
sizes where their padding and splitting can go wrong, and the two paths of f
and J (all signs known / any sign), against the oracle.

The mechanisms are synthetic ones around the warp's 32 lanes: fewer species
than lanes, one more or less than a full round, several rounds, and enough
reactions per species for targets of four pairs and more (two lanes each) and
for long species lists (a lane per chain).
"""
import os

import numpy as np
import pytest

from conftest import gpu_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

N_CELLS = 7


def _synthetic(tmp_path, n_species, n_rxn):
    from camp_b200.cells import make_cells
    from camp_b200.synth import load_synthetic

    mech, base = load_synthetic(str(tmp_path), n_species, n_rxn)
    return mech, make_cells(mech, N_CELLS, 41, conc_lo=1e-8, photo_base=base)


def _solver(mech, cells):
    from camp_b200.solver import Solver

    s = Solver(mech, cells.n_cells)
    s.initialize(abs_tol=np.full(mech.n_state_var, 1e-8), rel_tol=1e-4)
    s.set_photo_rates(cells.photo_rates)
    return s


SIZES = [(4, 6), (31, 40), (32, 40), (33, 45), (64, 70), (65, 70), (40, 160)]


@pytest.mark.parametrize("n_species,n_rxn", SIZES)
def test_small_mechanisms_f_and_jacobian(tmp_path, n_species, n_rxn):
    """f and J of the gathers against the oracle's to 1e-12 of production plus
    loss (an entry's two parts are signed, so by magnitude), as on the golden
    mechanisms."""
    from oracle.oracle import OracleModel

    mech, cells = _synthetic(tmp_path, n_species, n_rxn)
    s = _solver(mech, cells)
    f, p, l = s.eval_deriv(cells.state, cells.env, 60.0)
    j, jp, jl = s.eval_jac(cells.state, cells.env, 60.0)
    om = OracleModel(mech)
    for c in range(N_CELLS):
        env = om.rxn_env_row(cells.env[c], cells.photo_rates[c])
        of, _, _ = om.deriv(cells.state[c], env, 60.0)
        oj = om.jac(cells.state[c], env, 60.0)
        assert np.all(np.abs(f[c] - of) <= 1e-12 * (p[c] + l[c]))
        assert np.all(np.abs(j[c] - oj) <= 1e-12 * (np.abs(jp[c]) + np.abs(jl[c])))


@pytest.mark.parametrize("n_species,n_rxn", SIZES)
def test_small_mechanisms_solve(tmp_path, n_species, n_rxn):
    """The factorization and solves inside the integration: the oracle's
    outcomes, and against its tight solution the oracle's own accuracy (two
    runs at the same tolerances differ by their global errors), with the
    factors the other solve tests use."""
    from oracle.oracle import OracleModel

    mech, cells = _synthetic(tmp_path, n_species, n_rxn)
    s = _solver(mech, cells)
    assert s.kernel() == 0
    x = cells.state.copy()
    s.solve(x, cells.env, 0.0, 0.1)
    status = s.cell_stats()["status"]
    om, nt = OracleModel(mech), os.cpu_count() or 1

    def oracle(rtol, atol, max_steps):
        _, st, _, y = om.solve(cells.state.copy(), cells.env, cells.photo_rates, 0.0, 0.1, rtol,
                               np.full(mech.n_state_var, atol), max_steps=max_steps,
                               n_threads=nt)
        return st, y

    st, y = oracle(1e-4, 1e-8, 10000)
    tst, tight = oracle(1e-8, 1e-12, 200000)
    assert np.array_equal(status, st)
    rows = (st == 0) & (tst == 0)
    assert rows.any()
    dep = mech.dep_index()
    scale = 1e-4 * np.abs(tight[rows][:, dep]) + 1e-8
    eg = (np.abs(x - tight)[rows][:, dep] / scale).max(axis=1)
    ec = (np.abs(y - tight)[rows][:, dep] / scale).max(axis=1)
    assert np.median(eg) <= 2.0 * np.median(ec) + 1.0
    assert eg.max() <= 2.0 * ec.max() + 5.0


@pytest.mark.parametrize("name", ["cb05", "mod37", "mod37_soa", "mod37_aero", "mod37_shipped"])
def test_any_sign_path_matches_known_sign_path(name, request):
    """A species at -1e-31 ppm (above -SMALL, so f and J are defined) sends f
    and J down the term-by-term path; the same species at 0 takes the other.
    The terms differ by at most 1e-31 relative to ppm-sized concentrations, the
    sums' order by rounding, so the two agree to 1e-12 of production plus
    loss.  The species' own Jacobian row is left out: with its concentration
    the guard of its products changes sign."""
    from camp_b200.cells import make_cells

    mech = request.getfixturevalue(name)
    cells = make_cells(mech, N_CELLS, 43)
    dep = list(mech.dep_index())
    gas = [k for k, i in enumerate(dep) if "." not in mech.species[i]]
    zero, below = cells.state.copy(), cells.state.copy()
    moved = [gas[(7 * c + 3) % len(gas)] for c in range(N_CELLS)]
    for c, k in enumerate(moved):
        zero[c, dep[k]] = 0.0
        below[c, dep[k]] = -1e-31
    s = _solver(mech, cells)
    f0, p0, l0 = s.eval_deriv(zero, cells.env, 60.0)
    f1, _, _ = s.eval_deriv(below, cells.env, 60.0)
    assert np.all(np.abs(f1 - f0) <= 1e-12 * (p0 + l0) + 1e-25)
    j0, jp, jl = s.eval_jac(zero, cells.env, 60.0)
    j1, _, _ = s.eval_jac(below, cells.env, 60.0)
    rows = s.solver_jac()[1]
    other = rows[None, :] != np.asarray(moved)[:, None]
    assert np.all((np.abs(j1 - j0) <= 1e-12 * (np.abs(jp) + np.abs(jl)) + 1e-25)[other])
