"""Input validation: a bad entry at any place of a warp's rows (first and last
row of the warp, first and last entry, beside and in long rows, short and long
means) is refused with its own message, and good graphs are not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, degree, long_at, seed):
    rng = np.random.default_rng(seed)
    deg = np.full(n, degree)
    if long_at >= 0:
        deg[long_at] = 700   # past the limit of 512
    xadj = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    row = np.repeat(np.arange(n), deg)
    adj = ((row + 1 + rng.integers(0, n - 1, row.shape[0])) % n).astype(np.int32)   # never the row itself
    return xadj, adj, np.ones(adj.shape[0], np.int32), np.ones(n, np.int32), row


@pytest.mark.parametrize("n,degree,long_at", [(1000, 3, -1), (1000, 3, 40), (1000, 3, 31), (300, 70, -1), (40, 600, -1),
                                              (33, 2, 32)])
def test_bad_entry(pkg, handle, n, degree, long_at):
    xadj, adj, w, vw, row = _rows(n, degree, long_at, n + degree)
    handle.partition(xadj, adj, w, vw, 1)   # (one part: the rows are not symmetric)
    rows = sorted({0, 1, 30, 31, 32, n // 2, n - 1} & set(range(n)))
    for v in rows:
        for e in (xadj[v], xadj[v + 1] - 1):
            for arr, value, text in ((adj, n, "out of range"), (adj, -1, "out of range"), (adj, v, "self loop"),
                                     (w, -1, "negative weight")):
                bad = arr.copy()
                bad[e] = value
                with pytest.raises(pkg.GkwError, match=text):
                    handle.partition(xadj, bad if arr is adj else adj, bad if arr is w else w, vw, 1)
        bad = vw.copy()
        bad[v] = -1
        with pytest.raises(pkg.GkwError, match="negative weight"):
            handle.partition(xadj, adj, w, bad, 1)
        if v:
            bad = xadj.copy()
            bad[v] = xadj[v + 1] + 1
            with pytest.raises(pkg.GkwError, match="malformed xadj"):
                handle.partition(bad, adj, w, vw, 1)
