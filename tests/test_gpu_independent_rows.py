"""The independent-set test of the refinement candidates at its row lengths:
below, at and above eight entries a load (8), one sweep of a row (32) and the
limit to whole warps (64), gains positive nearly everywhere so that a warp
holds many rows.  Against the oracle, exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circulant(gen, n, degree, seed):
    """Every vertex with `degree` neighbours (even), ids shuffled."""
    rng = np.random.default_rng(seed)
    p = rng.permutation(n)
    i = np.arange(n)
    s = np.concatenate([p[i] for _ in range(degree // 2)])
    d = np.concatenate([p[(i + j + 1) % n] for j in range(degree // 2)])
    return gen.from_edges(n, s, d, rng.integers(1, 5, s.shape[0]), rng.integers(1, 4, n).astype(np.int32))


@pytest.mark.parametrize("degree", [2, 6, 8, 10, 30, 32, 34, 62, 64, 66])
@pytest.mark.parametrize("n", [70, 9000])
def test_rows(handle, orc, gen, degree, n):
    import torch
    g = _circulant(gen, n, degree, degree)
    k = 5
    dev = tuple(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (g.xadj, g.adjncy, g.adjwgt, g.vwgt))
    part = np.random.default_rng(n).integers(0, k, g.n).astype(np.int32)
    maxw = orc.max_part_weight(int(g.vwgt.astype(np.int64).sum()), k, 0.3)
    st = [part, np.zeros(n, np.int32), np.zeros(n, np.int32), part.copy(), np.ones(n, np.int32)]
    pw = orc.part_weights(g, part, k)
    ref = orc.refine(g, k, maxw, *st, pw, move_cap=1024)
    dv = [torch.from_numpy(a.copy()).cuda() for a in st]
    dpw = torch.from_numpy(pw.astype(np.int32)).cuda()
    rounds, moves = handle.refine(dev, k, maxw, 1024, *dv, dpw)
    assert (rounds, moves) == (ref["rounds"], ref["moves"])
    for t, key in zip(dv, ("part", "boundary", "gain", "target")):
        assert np.array_equal(t.cpu().numpy(), ref[key]), key
