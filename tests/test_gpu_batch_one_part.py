"""Graphs of one part in a union beside graphs whose halves do not fit one CTA.

A graph with k = 1 is never bisected, so the initial partition's member lists
keep its places as they were at the start through every depth, while the other
graph's row pass walks all places.  The dense graph is not coarsened (4000
vertices, k = 200, threshold 20k) and has about 120k entries a half at depth 1
and 30k a part at depth 3, above a CTA's shared memory; one one-part graph
coarsens, the other has no edges and does not.  Each graph's result is its lone
result, on memory that earlier batches have used."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dense(gen, n, deg, seed):
    rng = np.random.default_rng(seed)
    s = np.repeat(np.arange(n), deg // 2)
    return gen.from_edges(n, s, rng.integers(0, n, s.shape[0]), rng.integers(1, 9, s.shape[0]))


def _edgeless(gen, n):
    return gen.from_edges(n, np.zeros(0, np.int64), np.zeros(0, np.int64))


@pytest.mark.parametrize("order", [(0, 1, 2), (1, 0, 2), (2, 1, 0)])
def test_one_part_beside_large_halves(pkg, gen, order):
    graphs = [(_dense(gen, 4000, 60, 3), 200), (gen.delaunay(6000, 4), 1), (_edgeless(gen, 3000), 1)]
    graphs = [graphs[i] for i in order]
    gs, ks = [g for g, _ in graphs], [k for _, k in graphs]
    h = pkg.Handle(0)
    want = [h.partition(g.xadj, g.adjncy, g.adjwgt, g.vwgt, k)[:2] for g, k in graphs]
    h.close()
    x, a, w, vw, gp = pkg.concat_graphs(gs)
    fx, fa, fw, fvw, fgp = pkg.concat_graphs([gen.circuit(30000, seed=2, levels=60, hub_max=3000), gen.delaunay(9000, 5)])
    srv = pkg.Server(0)
    srv.partition_batch(fx, fa, fw, fvw, fgp, [64, 32])   # fills the pools with other values
    for _ in range(2):
        part, cuts, _ = srv.partition_batch(x, a, w, vw, gp, ks)
        for i, (p, c) in enumerate(want):
            assert cuts[i] == c
            assert np.array_equal(part[gp[i]:gp[i + 1]], p)
    srv.close()
