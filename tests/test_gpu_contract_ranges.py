"""Coarse rows beyond the first warp table on large levels, against the oracle:
through the 512-entry table, by direct accumulation over the row's own id range
(one window, its last id, four windows) and by hashing (five windows), and rows
that lose every entry to their own coarse vertex.  Integer work: exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WINDOW = 53248   # coarse ids of one window


def _blocks(gen, n, size, per, seed):
    """Edges inside blocks of `size` consecutive ids, `per` a vertex in every 8th block, else few."""
    rng = np.random.default_rng(seed)
    v = np.arange(n)
    cnt = np.where((v // size) % 8 == 0, per, 1)
    s = np.repeat(v, cnt)
    d = np.minimum(s // size * size + rng.integers(0, size, s.shape[0]), n - 1)
    return gen.from_edges(n, s, d, rng.integers(0, 9, s.shape[0]), rng.integers(1, 4, n).astype(np.int32))


def _spread(gen, n, fan, span, seed):
    """Hubs whose neighbours' ids span exactly `span`; the ring gives the first."""
    rng = np.random.default_rng(seed)
    hubs = np.arange(1, n - span, max(1, (n - span) // 30))[:30]
    s = np.repeat(hubs, fan + 1)
    d = np.concatenate([np.concatenate([[h + span - 2], h - 1 + rng.integers(0, span, fan)]) for h in hubs])
    ring = np.arange(n)
    return gen.from_edges(n, np.concatenate([s, ring]), np.concatenate([d, (ring + 1) % n]),
                          rng.integers(1, 9, s.shape[0] + n))


CASES = {
    "blocks_512": (lambda gen: _blocks(gen, 120000, 2000, 25, 1), 6),
    "blocks_over_512": (lambda gen: _blocks(gen, 120000, 2000, 50, 2), 20),
    "below_limit": (lambda gen: _blocks(gen, 90000, 2000, 25, 3), 6),
    "one_window": (lambda gen: _spread(gen, 330000, 900, WINDOW, 4), 1),
    "two_windows": (lambda gen: _spread(gen, 330000, 900, WINDOW + 1, 5), 1),
    "four_windows": (lambda gen: _spread(gen, 330000, 900, 4 * WINDOW, 6), 1),
    "five_windows": (lambda gen: _spread(gen, 330000, 900, 4 * WINDOW + 1, 7), 1),
    "five_windows_long": (lambda gen: _spread(gen, 330000, 9000, 4 * WINDOW + 1, 8), 1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_rows(handle, orc, gen, name):
    import torch
    make, cap = CASES[name]
    g = make(gen)
    cmap = (np.arange(g.n) // cap).astype(np.int32)
    nc = int(cmap[-1]) + 1
    dev = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))
    cx, ca, cw, cv = handle.contract(dev, torch.from_numpy(cmap).cuda(), nc)
    ox, oa, ow = orc.contract(g, cmap, nc)
    for got, want in ((cx, ox), (ca, oa), (cw, ow), (cv, orc.coarse_vwgt(g.vwgt, cmap, nc))):
        assert np.array_equal(got.cpu().numpy(), want)


def test_one_coarse_vertex_a_block(handle, orc, gen):
    """Whole blocks in one coarse vertex each: rows whose entries are all their own."""
    import torch
    n, size = 120000, 40
    rng = np.random.default_rng(9)
    s = np.repeat(np.arange(n), 10)
    d = s // size * size + rng.integers(0, size, s.shape[0])
    g = gen.from_edges(n, s, d, rng.integers(1, 9, s.shape[0]))
    cmap = (np.arange(n) // size).astype(np.int32)
    nc = n // size
    dev = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))
    cx, ca, cw, cv = handle.contract(dev, torch.from_numpy(cmap).cuda(), nc)
    assert int(cx.cpu()[-1]) == 0
    assert np.array_equal(cv.cpu().numpy(), orc.coarse_vwgt(g.vwgt, cmap, nc))
