"""Values of products, recurrences, eigen-pairs and Green's functions whose last bits matter: each sum in them runs in a
fixed order, and two kinds of results magnify a change of it.  A continued fraction of a state that is not the lowest of
its neighbouring sectors is not converged after 100 steps and depends on its start vector with a factor of up to 1e11
(a relative change of 1e-15 moves G by 1e-4); of a near-degenerate pair at the end of an FP32 solve's list one or the other
level is found.

``python tests/golden/make_solver_values.py OUT.npz`` (from the repository's root, on a GB300) stores them;
solver_values.npz was made before the operator's tiles, the Gram-Schmidt pass and the recurrences were rearranged.
"""
import os
import sys

import numpy as np

if __name__ == "__main__":
    sys.path.insert(0, os.getcwd())

from edlib_gb300 import ed, models

# model, sites, storage, sectors
PRODUCTS = [("siam", 12, "SRS", [(6, 6), (6, 4)]), ("siam", 10, "SRS", [(5, 4), (5, 2)]), ("kanamori", 8, "SRS", [(4, 4), (5, 6)]),
            ("kanamori", 12, "SRS", [(5, 4)]), ("ring", 8, "CRS", [(4, 4)]), ("siam", 10, "SOCRS", [(5, 4)]),
            ("kanamori", 7, "CRS", [(3, 3)])]
PAIRS = [("siam", 12, "SRS", (6, 6), "mixed"), ("siam", 9, "SRS", (4, 5), "fp64"), ("kanamori", 8, "SRS", (4, 4), "mixed"),
         ("kanamori", 7, "SRS", (3, 3), "fp64"), ("ring", 8, "CRS", (4, 4), "fp64"), ("siam", 10, "SOCRS", (5, 4), "fp32")]
# seeds of half-filled sectors of the 12-orbital impurity whose lowest state is not the model's
G_SEEDS = [325850717, 478558760, 33747223]
# a solve in which the last pair of a sector's list is near-degenerate with the next level
SOLVE_SEEDS = [184983849]


def model(kind, ns, seed, **more):
    if kind == "siam":
        params, data = models.random_siam(seed, ns - 1, U=3.0)
    elif kind == "kanamori":
        params, data = models.random_kanamori_siam(seed, nbath_per_orb=[(ns - 3 + 2 - m) // 3 for m in range(3)])
    else:
        params, data = {"NSITES": ns, "NSPINS": 2}, models.hubbard(models.ring_hopping(ns, 1.0), 4.0, 2.0)
    params.update({"arpack.NEV": 4, "lanc.BETA": 100.0, "lanc.NOMEGA": 32, "lanc.NLANC": 100, "lanc.BOLTZMANN_CUTOFF": 1e-12})
    params.update(more)
    return params, data


def hamiltonian(params, data, storage, precision, sector=None):
    if sector:
        params["arpack.SECTOR"] = 1
        data["sectors/values"] = np.array([sector], dtype=np.float64)
    p = ed.Params(params)
    ham = ed.Hamiltonian(p, data, storage=storage, precision=precision)
    ham.set_limits(0, 0)
    return p, ham


def some(x):
    """64 elements spread over a vector."""
    return np.asarray(x)[np.linspace(0, len(x) - 1, 64).astype(int)]


def products():
    for kind, ns, storage, sectors in PRODUCTS:
        for precision in ("fp32", "fp64"):
            _, ham = hamiltonian(*model(kind, ns, 5), storage, precision)
            for sec in sectors:
                v = np.random.default_rng(7).standard_normal(ham.storage.fill(*sec))
                v /= np.linalg.norm(v)
                name = "%s%d %s %s %d,%d" % (kind, ns, storage, precision, *sec)
                yield "product " + name, some(ham.storage.av(v))
                a, b, _ = ed.lanczos(ham, sec, v, 30)
                yield "recurrence " + name, np.stack([a[0], b[0][:30]])
            ham.close()


def pairs():
    for kind, ns, storage, sec, precision in PAIRS:
        _, ham = hamiltonian(*model(kind, ns, 5), storage, precision, sec)
        ham.diag()
        name = "%s%d %s %s %d,%d" % (kind, ns, storage, precision, *sec)
        yield "energies " + name, np.array([q.eigenvalue() for q in ham.eigenpairs()])
        if precision == "mixed":
            ed.refine_eigenpairs([ham], 100.0, 1e-12)
        yield "vector " + name, some(ham.eigenpairs()[0].eigenvector())
        ham.close()


def greens_functions():
    for seed in G_SEEDS:
        p, ham = hamiltonian(*model("siam", 12, seed), "SRS", "mixed", (6, 6))
        ham.diag()
        ed.refine_eigenpairs([ham], 100.0, 1e-12)
        g = ed.GreensFunction(p, ham)
        g.compute()
        yield "G %d" % seed, np.ascontiguousarray(g.G).view(np.float64)
        ham.close()


def solves():
    for seed in SOLVE_SEEDS:
        _, ham = hamiltonian(*model("siam", 12, seed, **{"arpack.NEV": 8}), "SRS", "mixed")
        ham.multiplicity_check = 2
        ham.diag()
        yield "spectrum %d" % seed, np.array([q.eigenvalue() for q in ham.eigenpairs()])
        ham.close()


GROUPS = {"products": products, "pairs": pairs, "greens_functions": greens_functions, "solves": solves}

if __name__ == "__main__":
    np.savez_compressed(sys.argv[1], **{k: v for f in GROUPS.values() for k, v in f()})
