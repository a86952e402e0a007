"""Device initial partition against the oracle at the edges of its layouts: the
one-CTA path (up to 1024 and 4096 members), the large path's tiers (rows in
shared memory, rows in L2, state by member, state in global memory), isolated
members, repeated entries, and weights that need 64-bit keys.  Integer work:
equality is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(g):
    import torch
    return tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))


def _sparse(gen, n, used, seed, wmax=8):
    """A random graph on `used` of n vertices (the others isolated), random
    weights, some vertex weights and edge weights zero."""
    rng = np.random.default_rng(seed)
    ids = np.sort(rng.choice(n, used, replace=False))
    s, d = rng.integers(0, used, 4 * used), rng.integers(0, used, 4 * used)
    w = rng.integers(0, wmax + 1, s.shape[0])
    return gen.from_edges(n, ids[s], ids[d], w, rng.integers(0, 5, n).astype(np.int32))


def _dense(gen, n, deg, seed):
    rng = np.random.default_rng(seed)
    s = np.repeat(np.arange(n), deg)
    d = np.minimum((rng.random(s.shape[0]) ** 3 * n).astype(np.int64), n - 1)   # hubs at the low ids
    return gen.from_edges(n, s, d, rng.integers(1, 9, s.shape[0]), rng.integers(1, 5, n).astype(np.int32))


def _scaled(g, gen, f):
    return gen.Csr(g.xadj, g.adjncy, (g.adjwgt.astype(np.int64) * f).astype(np.int32), g.vwgt)


def _repeated(g, gen):
    """Every entry listed twice (symmetric, with repeated neighbours)."""
    rep = np.repeat(np.arange(g.m), 2)
    return gen.Csr((2 * g.xadj).astype(np.int32), g.adjncy[rep].copy(), g.adjwgt[rep].copy(), g.vwgt)


CASES = {
    "one_word_block": lambda gen: gen.delaunay(32, 1),
    "small_1024": lambda gen: gen.delaunay(1024, 2),
    "small_1025": lambda gen: gen.delaunay(1025, 2),
    "rows_in_smem_4096": lambda gen: gen.delaunay(4096, 3),
    "rows_in_smem_4097": lambda gen: gen.delaunay(4097, 3),
    "rows_in_l2": lambda gen: _dense(gen, 3000, 60, 4),
    "rows_in_l2_two_levels": lambda gen: _dense(gen, 6000, 20, 5),
    "by_member": lambda gen: gen.delaunay(20000, 6),
    "isolated_small": lambda gen: _sparse(gen, 1500, 200, 7),
    "isolated_large": lambda gen: _sparse(gen, 9000, 1200, 8),
    "all_isolated": lambda gen: gen.from_edges(700, np.zeros(0, np.int64), np.zeros(0, np.int64)),
    "repeated_small": lambda gen: _repeated(gen.delaunay(900, 9), gen),
    "repeated_large": lambda gen: _repeated(gen.delaunay(5000, 9), gen),
    "index_does_not_fit": lambda gen: _scaled(gen.delaunay(2000, 10), gen, 1 << 22),
    "wide_small": lambda gen: _scaled(gen.delaunay(800, 11), gen, 1 << 26),
    "wide_large": lambda gen: _scaled(gen.delaunay(5000, 11), gen, 1 << 26),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_init_layouts(handle, orc, gen, name):
    g = CASES[name](gen)
    for k, trials in ((2, 8), (13, 8), (64, 3)) if g.n <= 10000 else ((2, 2),):
        p = handle.init_partition(_dev(g), k, seed=3, trials=trials).cpu().numpy()
        assert np.array_equal(p, orc.init_partition(g, k, seed=3, trials=trials)), (k, trials)


def test_init_state_in_global_memory(handle, orc, gen):
    g = gen.delaunay(70000, 12)   # above the map's 65535 members and the shared-memory words
    # heavy vertices in one corner of the id range end the oracle's growth early
    vw = np.ones(g.n, np.int32)
    vw[::97] = 400
    g = gen.Csr(g.xadj, g.adjncy, g.adjwgt, vw)
    p = handle.init_partition(_dev(g), 2, seed=1, trials=1).cpu().numpy()
    assert np.array_equal(p, orc.init_partition(g, 2, seed=1, trials=1))
