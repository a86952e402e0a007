"""Small coarsening levels against the oracle's whole run: one vertex up to the
one-CTA limit (14336) and just above, groups within the cap, of a few dozen,
of hundreds, of thousands and of the whole level, long candidate chains.
Every level's size, the rounds, the parts and the cut are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _stars(gen, n, leaves, seed):
    """Stars of about `leaves` leaves (one group each), ids shuffled, the hubs on a chain."""
    rng = np.random.default_rng(seed)
    hubs = np.arange(0, n, leaves + 1)
    leaf = np.setdiff1d(np.arange(n), hubs)
    s = np.concatenate([leaf, hubs[:-1]])
    d = np.concatenate([leaf // (leaves + 1) * (leaves + 1), hubs[1:]])
    w = np.concatenate([rng.integers(2, 9, leaf.shape[0]), np.ones(hubs.shape[0] - 1, np.int64)])
    p = rng.permutation(n)
    return gen.from_edges(n, p[s], p[d], w, rng.integers(1, 4, n).astype(np.int32))


def _chain(gen, n, seed):
    """A path of rising weights: one group, distances up to n - 1."""
    p = np.random.default_rng(seed).permutation(n)
    return gen.from_edges(n, p[:-1], p[1:], np.arange(1, n))


CASES = {
    "two": (lambda gen: gen.from_edges(2, np.array([0]), np.array([1])), 1),
    "no_edges": (lambda gen: gen.from_edges(70, np.zeros(0, np.int64), np.zeros(0, np.int64)), 2),
    "mesh_limit": (lambda gen: gen.delaunay(14336, 3), 4),
    "mesh_above": (lambda gen: gen.delaunay(14337, 4), 4),
    "pairs_and_sixes": (lambda gen: _stars(gen, 5000, 5, 5), 3),
    "groups_of_25": (lambda gen: _stars(gen, 14336, 24, 6), 3),
    "groups_of_90": (lambda gen: _stars(gen, 14000, 89, 7), 2),
    "groups_of_1000": (lambda gen: _stars(gen, 13007, 999, 8), 2),
    "groups_of_3000": (lambda gen: _stars(gen, 14336, 2999, 9), 2),
    "one_group": (lambda gen: _stars(gen, 14336, 14400, 10), 2),
    "chain": (lambda gen: _chain(gen, 3000, 11), 2),
    "dense_rows": (lambda gen: gen.circuit(9000, seed=12, levels=30, hub_max=3000), 4),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("cap", [1, 6, 40])
def test_levels(pkg, handle, orc, gen, name, cap):
    make, k = CASES[name]
    g = make(gen)

    def init(x, a, w, vw, kk):
        return ((np.arange(x.shape[0] - 1) * kk) // max(x.shape[0] - 1, 1)).astype(np.int32)

    ref, info = orc.partition(g, k, init=init, group_cap=cap, threshold_factor=2)
    o = pkg.default_options(enforce_balance=0, group_cap=cap, threshold_factor=2)
    part, cut, st = handle.partition(g.xadj, g.adjncy, g.adjwgt, g.vwgt, k, o, init=init)
    assert st["level_n"] == info["level_n"] and st["level_m"] == info["level_m"]
    assert st["uf_rounds"] == info["uf_launches"]
    assert np.array_equal(part, ref) and cut == info["cut"]
