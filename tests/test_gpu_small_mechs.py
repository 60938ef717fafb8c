"""The warp kernel on mechanisms whose LU, lists or yields lie at the edges of
its tables (tests/test_warp_tables.py asserts which rounds each one has).

An LU without L entries has no forward round, so the first round of the
triangular solves already scales by reciprocal pivots; a solve that left the
scaling out still converges where gamma * k < 1 and so shows as many more
steps, as step limits on stiff losses and as a total that is not conserved.
"""
import numpy as np
import pytest

import small_mechs
from conftest import gpu_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

RTOL, ATOL = 1e-4, 1e-8


def _run(mech, y, rates, t, precision, max_steps=10000):
    """(state, stats) of the library and (state, status, steps) of the oracle."""
    from camp_b200.solver import Solver
    from oracle.oracle import OracleModel

    n = y.shape[0]
    env = np.tile(np.array([298.0, 1.0e5]), (n, 1))
    atol = np.full(mech.n_state_var, ATOL)
    s = Solver(mech, n)
    s.initialize(abs_tol=atol, rel_tol=RTOL, max_steps=max_steps)
    s.set_precision(precision)
    assert s.kernel() == 0
    if rates.shape[1]:
        s.set_photo_rates(rates)
    x = y.copy()
    s.solve(x, env, 0.0, t)
    _, status, stats, o = OracleModel(mech).solve(y.copy(), env, rates, 0.0, t, RTOL, atol,
                                                  max_steps=max_steps)
    return x, s.cell_stats(), o, status, np.array([v.nst for v in stats])


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("t", [60.0, 900.0])
@pytest.mark.parametrize("n_species", [1, 2, 32, 33, 65])
def test_emission_and_first_order_loss(tmp_path, n_species, t, precision):
    """dy/dt = e - k y with k from 0.1 to 1e3 s-1 over the cells: the oracle's
    outcome, its step count to 20 %, and y = e/k + (y0 - e/k) exp(-k t) to ten
    error weights (the problem is contracting, so an error of each step's
    size, about a weight, is all that remains of the earlier ones)."""
    names = small_mechs.names_of(n_species)
    mech = small_mechs.mechanism(tmp_path, names, [
        {"type": kind, "species": x} for x in names for kind in ("EMISSION", "FIRST_ORDER_LOSS")])
    k = np.array([0.1, 1.0, 10.0, 100.0, 1000.0])[:, None] * np.linspace(0.5, 1.0, n_species)
    eq = np.linspace(0.2, 1.5, n_species)[None, :]
    rates = np.stack([k * eq, k], axis=2).reshape(len(k), -1)
    y = np.ones((len(k), n_species))
    x, st, o, status, nst = _run(mech, y, rates, t, precision)
    assert (status == 0).all() and (st["status"] == 0).all()
    assert (np.abs(st["nst"] - nst) <= 0.2 * nst).all(), (st["nst"], nst)
    expect = eq + (y - eq) * np.exp(-k * t)
    assert (np.abs(x - expect) <= 10.0 * (RTOL * expect + ATOL)).all()


@pytest.mark.parametrize("reverse", [False, True])
@pytest.mark.parametrize("n_species", [3, 40])
def test_chain_conserves_its_total(tmp_path, n_species, reverse):
    """X0 -> X1 -> ... in either state order, FP64: the columns of I - gamma*J
    add up to one, so a solve conserves the total to its own rounding: at
    most 1e-15 of the concentrations per species, iteration and pass."""
    mech = small_mechs.chain(tmp_path, n_species, reverse)
    y = np.random.default_rng(5).uniform(0.5, 1.0, (6, n_species))
    x, st, o, status, nst = _run(mech, y, np.zeros((6, 0)), 10.0, 0)
    assert (status == 0).all() and (st["status"] == 0).all()
    assert (np.abs(st["nst"] - nst) <= 0.2 * nst).all(), (st["nst"], nst)
    total = y.sum(axis=1)
    assert (np.abs(x.sum(axis=1) - total) <= 1e-15 * n_species * st["nni"] * total).all()


@pytest.mark.parametrize("negative", [False, True])
@pytest.mark.parametrize("n_species", [10, 41, 90, 400])
def test_hub_f_and_jacobian(tmp_path, n_species, negative):
    """Long lists and guarded terms: f and J against the oracle's to 1e-12 of
    production plus loss, as on the packed mechanisms.  Half of the cells
    hold species at 1e-9 ppm, where the guard drops terms."""
    from camp_b200.solver import Solver
    from oracle.oracle import OracleModel

    mech = small_mechs.hub(tmp_path, n_species, negative)
    n = 6
    rng = np.random.default_rng(8)
    y = rng.uniform(0.1, 1.0, (n, n_species))
    y[: n // 2] = np.where(rng.random((n // 2, n_species)) < 0.3, 1e-9, y[: n // 2])
    env = np.tile(np.array([298.0, 1.0e5]), (n, 1))
    s = Solver(mech, n)
    s.initialize(abs_tol=np.full(n_species, ATOL), rel_tol=RTOL)
    om = OracleModel(mech)
    for h in (0.01, 60.0):
        f, p, l = s.eval_deriv(y, env, h)
        j, jp, jl = s.eval_jac(y, env, h)
        for c in range(n):
            row = om.rxn_env_row(env[c], np.zeros(0))
            of, _, _ = om.deriv(y[c], row, h)
            oj = om.jac(y[c], row, h)
            assert np.all(np.abs(f[c] - of) <= 1e-12 * (p[c] + l[c]))
            assert np.all(np.abs(j[c] - oj) <= 1e-12 * (np.abs(jp[c]) + np.abs(jl[c])))


@pytest.mark.parametrize("n_species,n_rxn", [(15, 600), (30, 300), (10, 1000)])
def test_guarded_terms_f_and_jacobian(tmp_path, n_species, n_rxn):
    """Every product guarded: the gathers for any signs, staged; to the same
    bound as above.  Half of the cells hold a species below zero (above the
    smallest refused value) or at 1e-12 ppm."""
    from camp_b200.solver import Solver
    from oracle.oracle import OracleModel

    mech = small_mechs.dense_negative(tmp_path, n_species, n_rxn, 5)
    n = 6
    y = np.random.default_rng(9).uniform(0.1, 1.0, (n, n_species))
    y[0, 3], y[1, 1], y[2, :5] = -1e-31, 0.0, 1e-12
    env = np.tile(np.array([298.0, 1.0e5]), (n, 1))
    s = Solver(mech, n)
    s.initialize(abs_tol=np.full(n_species, ATOL), rel_tol=RTOL)
    om = OracleModel(mech)
    for h in (1e-5, 1.0):
        f, p, l = s.eval_deriv(y, env, h)
        j, jp, jl = s.eval_jac(y, env, h)
        for c in range(n):
            row = om.rxn_env_row(env[c], np.zeros(0))
            of, _, _ = om.deriv(y[c], row, h)
            oj = om.jac(y[c], row, h)
            assert np.all(np.abs(f[c] - of) <= 1e-12 * (p[c] + l[c]))
            assert np.all(np.abs(j[c] - oj) <= 1e-12 * (np.abs(jp[c]) + np.abs(jl[c])))


@pytest.mark.parametrize("precision", [0, 1])
def test_guarded_terms_solve(tmp_path, precision):
    """10 species, 1 000 reactions of guarded products: the oracle's outcomes
    and no concentration below zero (the guards make f jump, so the distance
    of two runs says nothing)."""
    mech = small_mechs.dense_negative(tmp_path, 10, 1000, 5)
    y = np.random.default_rng(9).uniform(0.1, 1.0, (6, 10))
    x, st, _, status, _ = _run(mech, y, np.zeros((6, 0)), 0.01, precision)
    assert (status == 0).all() and (st["status"] == 0).all()
    assert (x >= 0.0).all() and (x <= y + ATOL).all()


# cations, anions, modes: the programs' parts over the lanes (the first two), a
# lane per program
INORGANIC = [(2, 2, 1), (3, 3, 2), (4, 5, 1), (3, 3, 6), (4, 5, 2)]


def _inorganic(tmp_path, n_cation, n_anion, n_modes):
    from camp_b200.cells import make_cells

    mech = small_mechs.inorganic(tmp_path, n_cation, n_anion, n_modes)
    cells = make_cells(mech, 6, 7)
    cells.state[:, mech.species.index("H2O")] = [1e2, 2e3, 5e3, 1e4, 1.5e4, 2e4]  # ppm
    return mech, cells


@pytest.mark.parametrize("case", INORGANIC)
def test_ion_pairs_f_and_jacobian(tmp_path, case):
    """ZSR and PD-FiTE of a phase with many ion pairs: f to 1e-12 of production
    plus loss; J to 1e-10, as the parameter partials are sums of up to twenty
    signed terms that cancel before they enter the two parts."""
    from camp_b200.solver import Solver
    from oracle.oracle import OracleModel

    mech, cells = _inorganic(tmp_path, *case)
    s = Solver(mech, 6)
    s.initialize(abs_tol=np.full(mech.n_state_var, 1e-14), rel_tol=1e-6)
    s.set_photo_rates(cells.photo_rates)
    om = OracleModel(mech)
    f, p, l = s.eval_deriv(cells.state, cells.env, 1.0)
    j, jp, jl = s.eval_jac(cells.state, cells.env, 1.0)
    for c in range(6):
        row = om.rxn_env_row(cells.env[c], cells.photo_rates[c])
        of, _, _ = om.deriv(cells.state[c], row, 1.0)
        oj = om.jac(cells.state[c], row, 1.0)
        assert np.all(np.abs(f[c] - of) <= 1e-12 * (p[c] + l[c]))
        assert np.all(np.abs(j[c] - oj) <= 1e-10 * (np.abs(jp[c]) + np.abs(jl[c])) + 1e-300)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", INORGANIC)
def test_ion_pairs_solve(tmp_path, case, precision):
    """The oracle's outcomes and, in FP64, an error against its tight solution
    of at most ten times its own largest over the cells."""
    from camp_b200.solver import Solver
    from oracle.oracle import OracleModel

    mech, cells = _inorganic(tmp_path, *case)
    atol = np.full(mech.n_state_var, 1e-14)
    s = Solver(mech, 6)
    s.initialize(abs_tol=atol, rel_tol=1e-6)
    s.set_precision(precision)
    s.set_photo_rates(cells.photo_rates)
    x = cells.state.copy()
    s.solve(x, cells.env, 0.0, 10.0)
    om = OracleModel(mech)

    def oracle(rtol, atol):
        _, st, _, y = om.solve(cells.state.copy(), cells.env, cells.photo_rates, 0.0, 10.0, rtol,
                               np.full(mech.n_state_var, atol), max_steps=100000)
        return st, y

    status, o = oracle(1e-6, 1e-14)
    tstatus, tight = oracle(1e-9, 1e-17)
    assert (status == 0).all() and (tstatus == 0).all()
    assert (s.cell_stats()["status"] == 0).all()
    if precision == 0:
        dep = mech.dep_index()
        scale = 1e-6 * np.abs(tight) + 1e-14
        eg, ec = (np.max((np.abs(v - tight) / scale)[:, dep]) for v in (x, o))
        assert eg <= 10.0 * ec


@pytest.mark.parametrize("n_species", [41, 300])
def test_hub_solve(tmp_path, n_species):
    """Targets of hundreds of pairs (two lanes of each round in use) in the
    factorization and solves: the oracle's outcomes and values to a hundred
    times the tolerance (two runs at rtol 1e-6 each with its global error)."""
    from camp_b200.solver import Solver
    from oracle.oracle import OracleModel

    mech = small_mechs.hub(tmp_path, n_species)
    y = np.random.default_rng(6).uniform(0.1, 1.0, (6, n_species))
    env = np.tile(np.array([298.0, 1.0e5]), (6, 1))
    atol = np.full(n_species, 1e-12)
    s = Solver(mech, 6)
    s.initialize(abs_tol=atol, rel_tol=1e-6)
    x = y.copy()
    s.solve(x, env, 0.0, 10.0)
    _, status, _, o = OracleModel(mech).solve(y.copy(), env, np.zeros((6, 0)), 0.0, 10.0, 1e-6,
                                              atol)
    assert (status == 0).all() and (s.cell_stats()["status"] == 0).all()
    assert (np.abs(x - o) <= 1e-4 * np.abs(o) + 1e-10).all()


@pytest.mark.parametrize("h", [0.0, 1.0, -1.0])
def test_jacobian_guard_with_infinite_concentration(tmp_path, h):
    """The guard -rate * yield * h <= y is NaN for an infinite concentration at
    a step of zero and then drops the product, as in the oracle: equal values
    (small whole sums, no rounding)."""
    from camp_b200.solver import Solver
    from oracle.oracle import OracleModel

    mech = small_mechs.chain(tmp_path, 33, k=0.5)
    y = np.ones((4, 33))
    y[1, 0], y[2, 7], y[3, :] = np.inf, np.inf, 0.0
    env = np.tile(np.array([298.0, 1.0e5]), (4, 1))
    s = Solver(mech, 4)
    s.initialize(abs_tol=np.full(33, ATOL), rel_tol=RTOL)
    j = s.eval_jac(y, env, h)[0]
    om = OracleModel(mech)
    row = om.rxn_env_row(env[0], np.zeros(0))
    assert np.array_equal(j, np.stack([om.jac(y[c], row, h) for c in range(4)]))
