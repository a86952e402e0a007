"""Cut and part weights at every mean degree's lane count, with rows around the
whole-warp limit, against the oracle.  Integer work: exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,deg,hub", [(1, 0, 0), (33, 1, 0), (5000, 1, 0), (5000, 1, 129), (5000, 3, 4000),
                                       (4000, 12, 128), (900, 60, 700)])
@pytest.mark.parametrize("k", [1, 7, 5000])
def test_cut(handle, orc, gen, pkg, n, deg, hub, k):
    import torch
    rng = np.random.default_rng(n + deg + hub)
    s = np.concatenate([rng.integers(0, n, deg * n), np.zeros(hub, np.int64), np.full(hub, n // 2)])
    d = np.concatenate([rng.integers(0, n, deg * n), rng.choice(n, hub, replace=False), rng.choice(n, hub, replace=False)])
    g = gen.from_edges(n, s, d, rng.integers(0, 2**31 - 1, s.shape[0]), rng.integers(0, 2**31 - 1, n).astype(np.int32))
    dev = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))
    part = rng.integers(0, k, n).astype(np.int32)
    want = np.bincount(part, weights=None, minlength=k) * 0
    np.add.at(want, part, g.vwgt.astype(np.int64))
    for cut, pw in (handle.cut(dev, torch.from_numpy(part).cuda(), k),
                    pkg.cut_noalloc(dev, torch.from_numpy(part).cuda(), k)):
        assert cut == orc.cut(g, part)
        assert np.array_equal(pw, want)
