"""Small hand-made mechanisms at the edges of the warp kernel's tables: a
diagonal Jacobian, chains in either state order, a hub species in every
reaction, negative yields."""
import json
import os

from camp_b200.mechanism import load_mechanism


def mechanism(tmp_dir, names, rxns):
    """The mechanism of these species (in state order) and reactions, written
    as CAMP JSON input under tmp_dir and loaded."""
    species = {"camp-data": [{"name": n, "type": "CHEM_SPEC"} for n in names]}
    mech = {"camp-data": [{"name": "small", "type": "MECHANISM", "reactions": rxns}]}
    files = [os.path.join(str(tmp_dir), f) for f in ("small_species.json", "small_mech.json")]
    for f, obj in zip(files, (species, mech)):
        with open(f, "w") as fh:
            json.dump(obj, fh)
    return load_mechanism(files, "small")


def reaction(reactants, products, k=0.1):
    """A reaction of rate constant k; products maps names to yields."""
    return {"type": "ARRHENIUS", "A": k, "reactants": {r: {} for r in reactants},
            "products": {p: ({} if y == 1 else {"yield": y}) for p, y in products.items()}}


def names_of(n):
    return [f"X{i:03d}" for i in range(n)]


def diagonal(tmp_dir, n):
    """n species, each lost by itself: L and U without entries."""
    return mechanism(tmp_dir, names_of(n), [reaction([x], {}) for x in names_of(n)])


def chain(tmp_dir, n, reverse=False, k=0.1):
    """X0 -> X1 -> ... in state order, or with the products before their
    reactants (then L has no entries: ties in the pivot order go by index)."""
    names = names_of(n)
    o = names[::-1] if reverse else names
    return mechanism(tmp_dir, names, [reaction([a], {b: 1}, k) for a, b in zip(o, o[1:])])


def hub(tmp_dir, n, negative=False):
    """X0 reacts with every other species into X1: one long loss list, one
    long production list, rows and columns of the hub with n entries.  With
    negative yields each reaction also takes from a third species."""
    names = names_of(n)
    rxns = []
    for i, a in enumerate(names[2:]):
        products = {names[1]: 1}
        if negative:
            products[names[2 + (5 * i + 3) % (n - 2)]] = -0.25
        rxns.append(reaction([names[0], a], products))
    return mechanism(tmp_dir, names, rxns)


def dense_negative(tmp_dir, n, n_rxn, n_prod, seed=3):
    """Random bimolecular reactions whose products all have negative yields,
    so that every product term is guarded."""
    import numpy as np

    rng, names = np.random.default_rng(seed), names_of(n)
    rxns = []
    for _ in range(n_rxn):
        r = [names[i] for i in rng.choice(n, 2, replace=False)]
        rxns.append(reaction(r, {names[i]: -0.3 for i in rng.choice(n, n_prod, replace=False)}))
    return mechanism(tmp_dir, names, rxns)


def inorganic(tmp_dir, n_cation, n_anion, n_modes=1, n_interaction=None):
    """An aqueous phase in n_modes modes with every ion pair of the cations and
    anions: ZSR water, PD-FiTE activity coefficients of each pair (with every
    pair, or the first n_interaction, as interactions) and its equilibrium."""
    from camp_b200.aerosol import load_aerosol_mechanism

    def aerosol(name, **props):
        return dict({"name": name, "type": "CHEM_SPEC", "phase": "AEROSOL",
                     "density [kg m-3]": 1000.0}, **props)

    mw = "molecular weight [kg mol-1]"
    cations, anions = ([f"{k}{i}" for i in range(n)] for k, n in (("C", n_cation), ("A", n_anion)))
    pairs = [(c, a) for c in cations for a in anions]
    species = [{"name": "H2O", "type": "CHEM_SPEC"}]
    species += [aerosol(c, charge=1, **{mw: 0.018 + 0.002 * i}) for i, c in enumerate(cations)]
    species += [aerosol(a, charge=-1, **{mw: 0.06 + 0.01 * i}) for i, a in enumerate(anions)]
    for c, a in pairs:
        species.append(aerosol(f"{c}{a}", **{mw: 0.08}))
        species.append(aerosol(f"{c}-{a}", ions={c: {}, a: {}},
                               **{"tracer type": "ION_PAIR", mw: 0.08}))
    species.append(aerosol("H2O_aq", **{"tracer type": "CONSTANT", mw: 0.018}))
    phase = {"name": "aq", "type": "AERO_PHASE", "species": [s["name"] for s in species[1:]]}
    modes = {f"m{i}": {"type": "MODAL", "phases": ["aq"], "shape": "LOG_NORMAL",
                       "geometric mean diameter [m]": 1e-7, "geometric standard deviation": 1.6}
             for i in range(n_modes)}
    names = [f"{c}-{a}" for c, a in pairs]
    common = {"aerosol phase": "aq", "gas-phase water": "H2O", "aerosol-phase water": "H2O_aq"}
    water = dict(common, name="water", type="SUB_MODEL_ZSR_AEROSOL_WATER", **{"ion pairs": {
        f"{c}-{a}": {"type": "JACOBSON", "ions": {c: {}, a: {}}, "low RH": 0.3,
                     "Y_j": [1.0, -2.0 + 0.1 * i, 1.5, 0.1]} for i, (c, a) in enumerate(pairs)}})
    act = dict(common, name="activity", type="SUB_MODEL_PDFITE", **{"calculate for": {
        x: {"interactions": [{"ion pair": n, "min RH": 0.0, "max RH": 0.9 if i == 1 else 1.0,
                              "B": [0.1, -0.2, 0.05 + 0.01 * i, 0.01, -0.003]}
                             for i, n in enumerate(names[:n_interaction])]} for x in names}})
    rxns = [{"type": "AQUEOUS_EQUILIBRIUM", "aerosol phase": "aq", "aerosol-phase water": "H2O_aq",
             "reactants": {f"{c}{a}": {}}, "products": {c: {}, a: {}}, "A": 1e-3, "C": 300.0,
             "k_reverse": 0.1, "ion pair": f"{c}-{a}"} for c, a in pairs]
    doc = {"camp-data": species + [
        phase, {"name": "rep", "type": "AERO_REP_MODAL_BINNED_MASS", "modes/bins": modes}, water,
        act, {"name": "small", "type": "MECHANISM", "reactions": rxns}]}
    path = os.path.join(str(tmp_dir), "small_aero.json")
    with open(path, "w") as fh:
        json.dump(doc, fh)
    return load_aerosol_mechanism([path], name="small")
