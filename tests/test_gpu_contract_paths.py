"""Contraction through every kind of coarse row against the oracle: 16 lanes
per row (sparse levels), one warp per row with each table size, rows listed
from one to the next, and heavy rows by direct accumulation (few coarse ids,
or windows of many) and by the shared hash table.  Integer work: exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sparse(gen, n, per, seed):
    rng = np.random.default_rng(seed)
    s = rng.integers(0, n, int(per * n))
    d = np.clip(s + rng.integers(-40, 41, s.shape[0]), 0, n - 1)
    return gen.from_edges(n, s, d, rng.integers(0, 9, s.shape[0]), rng.integers(1, 4, n).astype(np.int32))


def _hubs(gen, n, per, hubs, fan, seed):
    rng = np.random.default_rng(seed)
    s = np.concatenate([rng.integers(0, n, int(per * n)), np.repeat(rng.choice(n, hubs, replace=False), fan)])
    d = rng.integers(0, n, s.shape[0])
    return gen.from_edges(n, s, d, rng.integers(1, 9, s.shape[0]))


CASES = {
    "tiny": lambda gen: _sparse(gen, 3, 1.0, 1),
    "short_rows": lambda gen: _sparse(gen, 50000, 1.1, 2),          # mean degree 2.2: 16 lanes
    "short_rows_with_hubs": lambda gen: _hubs(gen, 60000, 1.0, 30, 300, 3),
    "mesh": lambda gen: gen.delaunay(30000, 4),
    "grid27": lambda gen: gen.grid27(30, 31, 29),                    # rows of up to 156: 256 entries
    "degree_40": lambda gen: _sparse(gen, 20000, 20, 5),
    "degree_100": lambda gen: _hubs(gen, 4000, 50, 0, 0, 6),         # 512 entries, many heavier
    "dense_few_ids": lambda gen: _hubs(gen, 30000, 4, 40, 7000, 7),
    "many_ids_hash": lambda gen: _hubs(gen, 200000, 3, 60, 900, 8),   # more than 53248 coarse ids
    "many_ids_windows": lambda gen: _hubs(gen, 200000, 2, 5, 30000, 9),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("cap", [2, 6])
def test_contract_rows(handle, orc, gen, name, cap):
    import torch
    g = CASES[name](gen)
    rng = np.random.default_rng(cap)
    # groups of 1..cap vertices, near in id half of the time
    size = rng.integers(1, cap + 1, g.n)
    cmap = np.repeat(np.arange(g.n), size)[: g.n]
    nc = int(cmap[-1]) + 1
    far = rng.random(g.n) < 0.5
    idx = np.flatnonzero(far)
    cmap[idx] = cmap[rng.permutation(idx)]
    cmap = cmap.astype(np.int32)
    dev = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))
    cx, ca, cw, cv = handle.contract(dev, torch.from_numpy(cmap).cuda(), nc)
    ox, oa, ow = orc.contract(g, cmap, nc)
    for got, want in ((cx, ox), (ca, oa), (cw, ow), (cv, orc.coarse_vwgt(g.vwgt, cmap, nc))):
        assert np.array_equal(got.cpu().numpy(), want)
