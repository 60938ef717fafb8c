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
