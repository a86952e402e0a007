"""Rounds whose candidates exceed the move cap or put parts at risk: the ranked
selection and balance check of the level kernel against the oracle's sorted
rounds, from random partitions (thousands of candidates, tight caps).  Gains in
exact bins, in shared bins (weights up to 4000) and in one bucket (a star's
equal keys), ids in a narrow range, k at and above the check's part limit.
Integer work: equality is exact."""
import numpy as np
import pytest

from graphs import star_graph, weighted

pytestmark = pytest.mark.gpu


def _clustered(gen, n, seed):
    """Edges only among the last eighth of the ids: candidates share few buckets."""
    rng = np.random.default_rng(seed)
    lo = n - n // 8
    return gen.from_edges(n, rng.integers(lo, n, 3 * n), rng.integers(lo, n, 3 * n), rng.integers(1, 4, 3 * n))


CASES = {
    "mesh_unit": (lambda gen: gen.delaunay(40000, 1), (2, 64)),
    "mesh_weighted": (lambda gen: weighted(gen, gen.delaunay(30000, 2), 3, wmax=4000, vmax=9), (8, 1024)),
    "mesh_many_parts": (lambda gen: gen.delaunay(30000, 4), (1025, 1300)),
    "clustered_ids": (lambda gen: _clustered(gen, 40000, 5), (16, 100)),
    "star": (lambda gen: star_graph(gen, 9000), (2, 5)),
    "small": (lambda gen: gen.delaunay(40, 6), (2, 4)),
}


@pytest.mark.parametrize("cap", [1, 100, 1024, 2048])
@pytest.mark.parametrize("name", sorted(CASES))
def test_ranked_rounds(handle, orc, gen, name, cap):
    import torch
    make, ks = CASES[name]
    g = make(gen)
    if cap == 1 and g.n > 10000:
        pytest.skip("one move a round: tens of thousands of oracle rounds")
    dev = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))
    W = int(g.vwgt.astype(np.int64).sum())
    for k in ks:
        part = np.random.default_rng(k).integers(0, k, g.n).astype(np.int32)
        for eps in (0.03, 0.5):   # tight: most indices unbalanced; loose: most balanced
            st = [part, np.zeros(g.n, np.int32), np.zeros(g.n, np.int32), part.copy(), np.ones(g.n, np.int32)]
            pw = orc.part_weights(g, part, k)
            maxw = orc.max_part_weight(W, k, eps)
            ref = orc.refine(g, k, maxw, *st, pw, move_cap=cap)
            dv = [torch.from_numpy(a.copy()).cuda() for a in st]
            dpw = torch.from_numpy(pw.astype(np.int32)).cuda()
            rounds, moves = handle.refine(dev, k, maxw, cap, *dv, dpw)
            assert (rounds, moves) == (ref["rounds"], ref["moves"]), (k, eps)
            for t, key in zip(dv, ("part", "boundary", "gain", "target")):
                assert np.array_equal(t.cpu().numpy(), ref[key]), (k, eps, key)
            assert np.array_equal(dpw.cpu().numpy().astype(np.int64), ref["pw"]), (k, eps)


def _rows(gen, n, hubs, fan, seed):
    """A sparse graph with `hubs` rows of about `fan` entries, zero weights included."""
    rng = np.random.default_rng(seed)
    s = np.concatenate([rng.integers(0, n, 2 * n), np.repeat(rng.choice(n, hubs, replace=False), fan)])
    d = rng.integers(0, n, s.shape[0])
    return gen.from_edges(n, s, d, rng.integers(0, 6, s.shape[0]), rng.integers(1, 4, n).astype(np.int32))


@pytest.mark.parametrize("fan", [40, 80, 300, 1500, 2600])   # around 64 and 2048 entries, and the hubs' list
@pytest.mark.parametrize("k", [3, 64, 700])
def test_long_rows(handle, orc, gen, fan, k):
    """Gain updates, rounds and balance rounds over long rows, against the oracle."""
    import torch
    g = _rows(gen, 6000, 400 if fan < 1000 else 150, fan, fan)
    dev = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))
    part = np.random.default_rng(k).integers(0, k, g.n).astype(np.int32)
    W = int(g.vwgt.astype(np.int64).sum())
    zeros = np.zeros(g.n, np.int32)
    # refinement rounds from a random partition
    st = [part, zeros.copy(), zeros.copy(), part.copy(), np.ones(g.n, np.int32)]
    pw = orc.part_weights(g, part, k)
    maxw = orc.max_part_weight(W, k)
    ref = orc.refine(g, k, maxw, *st, pw, move_cap=1024)
    dv = [torch.from_numpy(a.copy()).cuda() for a in st]
    dpw = torch.from_numpy(pw.astype(np.int32)).cuda()
    assert handle.refine(dev, k, maxw, 1024, *dv, dpw) == (ref["rounds"], ref["moves"])
    for t, key in zip(dv, ("part", "boundary", "gain", "target")):
        assert np.array_equal(t.cpu().numpy(), ref[key]), key
    # balance rounds from an overloaded partition
    over = part.copy()
    over[np.random.default_rng(1).random(g.n) < 0.3] = k - 1
    src = np.repeat(np.arange(g.n), np.diff(g.xadj))
    bnd = np.zeros(g.n, np.int32)
    np.logical_or.at(bnd, src, over[src] != over[g.adjncy])
    pw = orc.part_weights(g, over, k)
    cap = orc.balance_cap(W, k)
    ref = orc.balance(g, k, cap, over, bnd, zeros, over, pw, move_cap=1024)
    dv = [torch.from_numpy(a.copy()).cuda() for a in (over, bnd, zeros, over)]
    dpw = torch.from_numpy(pw.astype(np.int32)).cuda()
    handle.balance(dev, k, cap, 1024, *dv, dpw)
    for t, key in zip(dv, ("part", "boundary", "gain", "target")):
        assert np.array_equal(t.cpu().numpy(), ref[key]), key
