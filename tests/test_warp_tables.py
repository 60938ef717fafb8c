"""Tables of the warp-per-cell kernel, checked on the CPU.

The warp kernel (camp_b200/csrc/solve.cu) factors I - gamma*J by pivot levels
and solves with the factors in rounds of 32 targets, each round a table row
with one record per lane, the same number of pairs in every lane and, for long
targets, two lanes per target; f and J are gathered in rounds of eight items
with a lane per chain of sums and rounds of 32 items with a lane per item.
These tests replay the rounds in numpy on the tables the library builds (every
index the kernel reads comes from them): the factors and the solution against
dense linear algebra, for a random matrix with the mechanism's LU pattern, and
the gathers' sums against the term lists of the path for any signs.  Among the
mechanisms are those whose L or U has no entries, whose targets are long and
whose terms are guarded, and the tests assert that their tables have such
rounds.
"""
import ctypes as C
import tempfile

import numpy as np
import pytest

import small_mechs

LANES = 32
GATHER = "n_a n_b n_neg zero a_rec a_ent b_hdr b_id b_ent neg".split()


class Gather(C.Structure):
    _fields_ = [(f, C.c_int) for f in GATHER]


class BlobOff(C.Structure):
    """The header of the tables (blob.hpp)."""
    _fields_ = (
        [(f, C.c_int) for f in (
            "bytes stage_bytes seq_bytes n n_rxn n_part n_jac n_lu n_coef n_fsplit n_fscratch "
            "n_plev any_sign rx_word rx_vptr coef fg_ent fg_unit fg_lane fg_split").split()]
        + [("g", Gather * 2), ("self", C.c_ulonglong)]
        + [(f, C.c_int) for f in (
            "jg_w0 jg_w1 jg_ptr jg_mid jg_lupos jg_row jg_lane jg_slots j_csc jg_slot lu_iperm "
            "lu_diag lu_src fl_hdr fs_rec fb_rec fb_ext n_fwd n_bwd sv_rec sv_ext lu_rowptr "
            "lu_col upd_ptr upd dep_state atol n_simpol n_keff n_rates n_part_all si_rec si_elem "
            "si_ef n_aq aq_rec aq_sp aq_sm aq_cp aq_cpm aq_sim has_ug jg_umid n_cv n_pj sm_keff "
            "sm_rec sm_int sm_flt sm_state n_smi sm_item sm_scr n_smp sm_pel sm_pq n_sms").split()]
        + [("scr0", C.c_int * 2), ("scr_end", C.c_int * 2)])


class Tables:
    def __init__(self, mech):
        from camp_b200.solver import Solver

        s = Solver(mech, 4)
        s.build_sparsity_only()
        self.raw = s.warp_tables()
        self.o = o = BlobOff.from_buffer_copy(self.raw)
        assert o.bytes == len(self.raw)  # the header above is the library's
        n = o.n
        self.iperm = self.arr(o.lu_iperm, np.uint16, n)
        self.diag = self.arr(o.lu_diag, np.uint16, n)
        self.rowptr = self.arr(o.lu_rowptr, np.uint16, n + 1)
        self.col = self.arr(o.lu_col, np.uint16, o.n_lu)
        self.coef = np.frombuffer(self.raw, np.float64, o.n_coef, o.coef)

    def arr(self, at, dtype, count):
        return np.frombuffer(self.raw, dtype, int(count), int(at)).astype(np.int64)

    def words(self, at):
        """uint32 words from `at` to the end of the tables."""
        return self.arr(at, np.uint32, (len(self.raw) - at) // 4)


def pair_round(rec, ext, A, X, spare):
    """One round of targets X[t] -= sum A[a] X[x]: returns (targets, sums,
    words of ext used).  A and X end with their spare slot, which stays 0."""
    w0, w1 = rec[0::2], rec[1::2]
    a, x = w0 & 0xFFFF, w0 >> 16
    cnt = w1 >> 16
    assert (cnt == cnt[0]).all()
    two = bool(cnt[0] & 0x8000)
    c, row = (cnt[0] & 0x3FF, cnt[0] >> 9 & 62) if two else (cnt[0], LANES)
    lanes = np.arange(LANES)
    tgt = w1 & 0x7FFF if spare < 0x8000 else w1 & 0xFFFF
    s = X[tgt] - A[a] * X[x]
    for k in range(c - 1):
        q = ext[row * k + lanes]  # idle lanes read on
        s = s - A[q & 0xFFFF] * X[q >> 16]
    if two:
        s = np.where((lanes % 2 == 0) & (lanes < row), s + s[lanes ^ 1], 0.0)
        assert (tgt[1::2] == spare).all() and (tgt[row:] == spare).all()
    assert (s[tgt == spare] == 0.0).all()
    real = tgt[tgt != spare]
    assert len(np.unique(real)) == len(real)
    return tgt, s, int(row * (c - 1))


def factor(t, LU):
    """dev_form_factor's rounds on LU (with its spare slot, in place);
    returns the reciprocal pivots."""
    o = t.o
    hdr = t.arr(o.fl_hdr, np.uint16, 2 * o.n_plev)
    fs, rec, ext = t.words(o.fs_rec), t.words(o.fb_rec), t.words(o.fb_ext)
    dinv = np.full(o.n, np.nan)
    f0 = r = e = 0
    for lv in range(o.n_plev):
        f1, rounds = hdr[2 * lv], hdr[2 * lv + 1]
        w0, w1 = fs[2 * f0:2 * f1:2], fs[2 * f0 + 1:2 * f1:2]
        f0 = f1
        d = 1.0 / LU[w0 >> 16]
        pos, at = w0 & 0xFFFF, w1 & 0x8000 != 0
        assert not set(pos.tolist()) & set((w0 >> 16).tolist())
        LU[pos[pos != o.n_lu]] *= d[pos != o.n_lu]
        assert np.isnan(dinv[w1[at] & 0x7FFF]).all()  # each stored once
        dinv[w1[at] & 0x7FFF] = d[at]
        for _ in range(rounds):
            tgt, s, used = pair_round(rec[64 * r:64 * r + 64], ext[e:], LU, LU, o.n_lu)
            LU[tgt] = s
            r, e = r + 1, e + used
    assert not np.isnan(dinv).any()
    return dinv


def solve(t, LU, dinv, b):
    """dev_lsolve's rounds: b (dependent order) -> M^{-1} b."""
    o = t.o
    rec, ext = t.words(o.sv_rec), t.words(o.sv_ext)
    z = np.zeros(o.n + 1)
    z[t.iperm] = b
    e, finished = 0, []
    for r in range(o.n_fwd + o.n_bwd):
        w = rec[64 * r:64 * r + 64]
        tgt, s, used = pair_round(w, ext[e:], LU, z, o.n)
        finish = w[1::2] & 0x8000 != 0
        assert r >= max(1, o.n_fwd) or not finish.any()  # the first takes no reciprocal
        finished += tgt[finish].tolist()
        z[tgt] = np.where(finish, s * dinv[np.minimum(tgt, o.n - 1)], s)
        e += used
    assert sorted(finished) == list(range(o.n))  # each pivot once
    return z[t.iperm]


def sums(t, k, src):
    """Production and loss sums per item id of the f (k = 0) or J (k = 1)
    gather, from its chain and item rounds."""
    o, g = t.o, t.o.g[k]
    src = np.append(src, np.zeros(1 + g.n_neg))  # the zero and the guarded terms
    assert len(src) == g.zero + 1 + g.n_neg
    neg = t.arr(g.neg, np.uint32, 2 * g.n_neg)[0::2]
    src[g.zero + 1:] = src[neg & 0xFFFF] * t.coef[neg >> 16] * (-1.0 if k == 0 else 1.0)
    assert not o.any_sign
    P, L = {}, {}

    def add(word, p, l):
        i = int(word) & 0xFFFF
        if i != 0xFFFF:
            P[i], L[i] = P.get(i, 0.0) + p, L.get(i, 0.0) + l

    rec, ent = t.words(g.a_rec), t.words(g.a_ent)
    for r in range(g.n_a):
        for item in range(8):
            v = []
            for c in range(4):
                w0, w1 = rec[2 * (LANES * r + 4 * item + c):][:2]
                q = ent[w0 & 0xFFFF:][:w0 >> 16]
                v.append((src[q & 0xFFFF] * t.coef[q >> 16]).sum())
            add(w1, v[2] + v[3], v[0] + v[1])
    hdr, at = t.words(g.b_hdr), 0
    ids = t.words(g.b_id) if k == 0 else t.arr(g.b_id, np.uint16, LANES * g.n_b)
    ent = t.words(g.b_ent)
    for r in range(g.n_b):
        n_loss, n_prod, n_lead = hdr[2 * r] & 0xFFFF, hdr[2 * r] >> 16, hdr[2 * r + 1]
        rows = ent[at:at + LANES * (n_lead + n_loss + n_prod)].reshape(-1, LANES)
        at += rows.size
        lead, loss, prod = np.split(rows, [n_lead, n_lead + n_loss])
        p = src[lead & 0xFFFF].sum(0) + (src[prod & 0xFFFF] * t.coef[prod >> 16]).sum(0)
        l = src[loss & 0xFFFF].sum(0) + src[loss >> 16].sum(0)
        for lane in range(LANES):
            add(ids[LANES * r + lane], p[lane], l[lane])
    return P, L


def check_factor_and_solve(t, seed):
    n, n_lu = t.o.n, t.o.n_lu
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))  # in pivot order
    for i in range(n):
        A[i, t.col[t.rowptr[i]:t.rowptr[i + 1]]] = rng.uniform(-1.0, 1.0)
    A *= rng.uniform(0.5, 1.0, (n, n))
    A[np.arange(n), np.arange(n)] = n + rng.uniform(0.0, 50.0, n)
    LU = np.zeros(n_lu + 1)
    for i in range(n):
        LU[t.rowptr[i]:t.rowptr[i + 1]] = A[i, t.col[t.rowptr[i]:t.rowptr[i + 1]]]
    dinv = factor(t, LU)
    L, U = np.eye(n), np.zeros((n, n))
    for i in range(n):
        for q in range(t.rowptr[i], t.rowptr[i + 1]):
            (L if t.col[q] < i else U)[i, t.col[q]] = LU[q]
    assert np.allclose(L @ U, A, rtol=1e-12, atol=1e-12 * n)
    assert np.allclose(dinv, 1.0 / np.diag(U), rtol=1e-14)
    b = rng.uniform(-1.0, 1.0, n)
    x = solve(t, LU, dinv, b)
    assert np.allclose(A[np.ix_(t.iperm, t.iperm)] @ x, b, rtol=1e-10, atol=1e-12)


def check_gathers(t, seed):
    o = t.o
    rng = np.random.default_rng(seed)
    # f: rates, then the computed species; units of the path for any signs
    src = rng.uniform(0.0, 1.0, o.g[0].zero)
    n_units = int(t.arr(o.fg_lane, np.uint16, 33)[32])
    ent = t.words(o.fg_ent)
    P, L = np.zeros(o.n), np.zeros(o.n)
    for sp, b, m1, m2, e, *_ in t.arr(o.fg_unit, np.uint16, 8 * n_units).reshape(-1, 8):
        c = t.coef[(ent[b:e] >> 16) & 0x7FFF] * src[ent[b:e] & 0xFFFF]
        L[sp] += src[ent[b:m1] & 0xFFFF].sum() - c[m2 - b:].sum()
        P[sp] += c[m1 - b:m2 - b].sum()
    p, l = sums(t, 0, src)
    for i in range(o.n):
        assert abs(p.get(i, 0.0) - P[i]) <= 1e-13 * (P[i] + L[i])
        assert abs(l.get(i, 0.0) - L[i]) <= 1e-13 * (P[i] + L[i])
    # J: partials, by CSC entry
    src = rng.uniform(0.0, 1.0, o.g[1].zero)
    p, l = sums(t, 1, src)
    slot = t.arr(o.jg_slot, np.uint16, o.n_jac)
    assert sorted(slot) == list(range(o.n_jac)) and sorted(p) == list(range(o.n_jac))
    w0 = t.words(o.jg_w0)
    ptr = t.arr(o.jg_ptr, np.uint16, o.n_jac + 1)
    umid, mid = (t.arr(a, np.uint16, o.n_jac) for a in (o.jg_umid, o.jg_mid))
    for e in range(o.n_jac):
        v = src[w0[ptr[e]:ptr[e + 1]] & 0xFFFF]
        c = v * t.coef[w0[ptr[e]:ptr[e + 1]] >> 16]
        u, m = umid[e] - ptr[e], mid[e] - ptr[e]
        P, L = v[:u].sum() + c[m:].sum(), v[u:m].sum()
        scale = 1e-13 * (v[:m].sum() + np.abs(c[m:]).sum())
        assert abs(p[slot[e]] - P) <= scale and abs(l[slot[e]] - L) <= scale


def empty_forward(t):
    """Whether the forward rounds are a single one without targets."""
    w = t.words(t.o.sv_rec)[1:64 * t.o.n_fwd:2]
    return t.o.n_fwd == 1 and (w & 0x7FFF == t.o.n).all()


@pytest.mark.parametrize("which", ["cb05", "mod37", "mod37_soa", "mod37_aero", "mod37_shipped"])
def test_packed_mechanisms(request, which):
    t = Tables(request.getfixturevalue(which))
    check_factor_and_solve(t, 3)
    check_gathers(t, 4)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65])
def test_diagonal_system(tmp_path, n):
    """Neither L nor U has entries: an empty forward round, since the solve's
    first round takes no reciprocal pivots, and ceil(n / 32) backward ones."""
    t = Tables(small_mechs.diagonal(tmp_path, n))
    assert t.o.n_lu == n and t.o.n_bwd == (n + 31) // 32
    assert empty_forward(t)
    check_factor_and_solve(t, 5)
    check_gathers(t, 6)


@pytest.mark.parametrize("kind", ["EMISSION", "FIRST_ORDER_LOSS", "WET_DEPOSITION"])
def test_host_rate_systems(kind):
    from conftest import species_rate_case

    t = Tables(species_rate_case(kind)[0])
    assert empty_forward(t)
    check_factor_and_solve(t, 5)
    check_gathers(t, 6)


@pytest.mark.parametrize("n", [3, 40])
@pytest.mark.parametrize("reverse", [False, True])
def test_chain(tmp_path, n, reverse):
    t = Tables(small_mechs.chain(tmp_path, n, reverse))
    assert empty_forward(t) == reverse
    check_factor_and_solve(t, 7)
    check_gathers(t, 8)


@pytest.mark.parametrize("negative", [False, True])
@pytest.mark.parametrize("n", [10, 41, 90, 300])
def test_hub(tmp_path, n, negative):
    """Long lists (a lane per chain), long targets (two lanes each), guarded
    terms."""
    t = Tables(small_mechs.hub(tmp_path, n, negative))
    g = t.o.g
    assert n < 41 or g[1].n_a > 0
    assert (g[0].n_neg > 0) == negative and (g[1].n_neg > 0) == negative
    cnt = t.words(t.o.sv_rec)[1:64 * (t.o.n_fwd + t.o.n_bwd):64] >> 16
    two = cnt[cnt & 0x8000 != 0]
    assert len(two)
    # a row of further pairs has a word per lane in use: few for the hub's own
    if n == 300:
        assert (two & 0x3FF).max() > 64 and ((two[(two & 0x3FF) > 64] >> 9 & 62) <= 4).all()
    check_factor_and_solve(t, 9)
    check_gathers(t, 10)


@pytest.mark.parametrize("n_species,n_rxn", [(4, 6), (33, 45), (65, 70), (40, 160)])
def test_synthetic(n_species, n_rxn):
    from camp_b200.synth import load_synthetic

    with tempfile.TemporaryDirectory() as d:
        mech, _ = load_synthetic(d, n_species, n_rxn)
    t = Tables(mech)
    check_factor_and_solve(t, 11)
    check_gathers(t, 12)


@pytest.mark.parametrize("n_species,n_rxn,any_sign", [(15, 600, 1), (30, 300, 1), (10, 1000, 1),
                                                       (20, 20, 0)])
def test_guarded_terms_take_no_cells(tmp_path, n_species, n_rxn, any_sign):
    """A guarded term would take a slot of every cell's slab: where that costs
    cells, the gathers for any signs are staged and the others empty."""
    t = Tables(small_mechs.dense_negative(tmp_path, n_species, n_rxn, 5))
    o = t.o
    assert o.any_sign == any_sign
    for k in range(2):
        assert (o.g[k].n_neg == 0 and o.g[k].n_a + o.g[k].n_b == 0) == bool(any_sign)
    for at in (o.fg_ent, o.fg_unit, o.fg_lane, o.jg_slot, o.jg_w0, o.jg_w1, o.jg_ptr, o.jg_umid):
        assert (at < o.stage_bytes) == bool(any_sign)
    check_factor_and_solve(t, 13)


@pytest.mark.parametrize("n_cation,n_anion,n_modes,parts", [
    (2, 2, 1, True), (2, 2, 8, True), (3, 3, 2, True), (4, 5, 1, False), (3, 3, 6, False)])
def test_ion_pairs(tmp_path, n_cation, n_anion, n_modes, parts):
    """The parts of the sub-models' programs are left out where their tables
    and scratch would cost cells, and their tables grow with the programs: an
    item of 16 bytes per interaction and two list entries per ion pair."""
    t = Tables(small_mechs.inorganic(tmp_path, n_cation, n_anion, n_modes))
    o, n_pair = t.o, n_cation * n_anion
    assert (o.n_smi > 0) == parts
    if parts:
        n_act = n_modes * n_pair
        assert o.n_cv == n_act + n_modes
        assert o.n_smi == n_act * n_pair + 2 * n_modes * n_pair
        assert o.n_sms == n_act * (3 * n_pair + 2) + n_modes * (7 + 2) * n_pair
        over = o.n_sms <= min(o.n_rates, o.n_part_all)
        ends = [g.zero + 1 + g.n_neg for g in o.g]
        assert list(o.scr0) == ([0, 0] if over else ends)
        assert list(o.scr_end) == (ends if over else [e + o.n_sms for e in ends])
        pel = t.arr(o.sm_pel, np.uint32, 2 * o.n_smp)
        assert o.n_smp == n_act * (1 + n_cation + n_anion)
        # every pair but the coefficient's own, against its cation and its anion
        assert (pel[1::2] >> 16).sum() == n_act * 2 * (n_pair - 1)
    check_factor_and_solve(t, 14)
    check_gathers(t, 15)
