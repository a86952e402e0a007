"""Rows that end at the last places an int32 CSR can have (2^31 - 2 entries).

A strided walk's next place passes 2^31 there, so every kernel that walks rows
is run on the last rows of two circulant graphs (row v: v + o mod n for the
offsets o, without the edge between the last two vertices): 4M rows of 512
entries and 65536 rows of 32768.  Unit weights; expected values of the last
rows are computed from the adjacency itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NEEDED = 100 << 30   # 17 GB of arrays, as much again for a contraction's output and scratch


def _circulant(torch, n, deg):
    half = deg // 2
    off = torch.cat([torch.arange(-half, 0), torch.arange(1, half + 1)]).cuda()
    adj = torch.empty(n * deg, dtype=torch.int32, device="cuda")
    rows = adj.view(n, deg)
    step = max(1, (1 << 27) // deg)
    for v in range(0, n, step):
        rows[v:v + step] = ((torch.arange(v, v + step, device="cuda")[:, None] + off) % n).to(torch.int32)
    last = [((v + off) % n).to(torch.int32) for v in (n - 2, n - 1)]
    last = torch.cat([last[0][last[0] != n - 1], last[1][last[1] != n - 2]])
    m = n * deg - 2
    adj[(n - 2) * deg:m] = last
    x = torch.arange(n + 1, device="cuda") * deg
    x[n - 1] -= 1
    x[n] = m
    assert m == 2 ** 31 - 2
    g = (x.to(torch.int32), adj[:m], torch.ones(m, dtype=torch.int32, device="cuda"),
         torch.ones(n, dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return g


@pytest.fixture(scope="module", params=[(1 << 22, 512), (1 << 16, 32768)], ids=["rows_512", "rows_32768"])
def graph(request):
    import torch
    if torch.cuda.mem_get_info()[0] < NEEDED:
        pytest.skip("needs 100 GB of device memory")
    g = _circulant(torch, *request.param)
    yield g
    del g
    torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def h(pkg):
    handle = pkg.Handle(0)
    yield handle
    handle.close()


def _row(g, v):
    b, e = int(g[0][v]), int(g[0][v + 1])
    return g[1][b:e].cpu().numpy()


def test_validation_reads_the_last_entry(graph, h, pkg):
    import torch
    n, m = graph[3].numel(), graph[1].numel()
    part = torch.empty(n, dtype=torch.int32, device="cuda")
    keep = int(graph[1][m - 1])
    for bad, text in ((n - 1, "self"), (n, "out of range"), (-1, "out of range")):
        graph[1][m - 1] = bad
        torch.cuda.synchronize()
        with pytest.raises(pkg.GkwError, match=text):
            h.partition_device(*graph, 4, part)
    graph[1][m - 1] = keep
    graph[2][m - 1] = -1
    torch.cuda.synchronize()
    with pytest.raises(pkg.GkwError, match="negative"):
        h.partition_device(*graph, 4, part)
    graph[2][m - 1] = 1
    torch.cuda.synchronize()


def test_match(graph, h):
    n = graph[3].numel()
    cand = h.match(graph).cpu().numpy()
    for v in list(range(n - 40, n)) + [0, 1, n // 2]:
        a = _row(graph, v)
        short = a[(a == n - 1) | (a == n - 2)]   # the smaller degree first, then the place in the row
        assert cand[v] == (short[0] if short.size else a[0]), v


def test_cut(graph, h):
    import torch
    n = graph[3].numel()
    part = (torch.arange(n, device="cuda") * 5 // n).to(torch.int32)
    want = 0
    rows = max(1, (1 << 27) // (graph[1].numel() // n))
    for v in range(0, n, rows):
        b, e = int(graph[0][v]), int(graph[0][min(v + rows, n)])
        src = torch.repeat_interleave(torch.arange(v, min(v + rows, n), device="cuda"),
                                      (graph[0][v + 1:v + rows + 1] - graph[0][v:v + rows][:n - v]).long())
        dst = graph[1][b:e].long()
        want += int(((dst > src) & (part[dst] != part[src])).sum())
    torch.cuda.synchronize()
    cut, pw = h.cut(graph, part, 5)
    assert cut == want and pw.tolist() == torch.bincount(part).tolist()


def test_update_and_refine_and_balance(graph, h):
    """Part 1 is the first quarter: only the last vertex has a positive gain,
    and the caps leave room for one move."""
    import torch
    n = graph[3].numel()
    ids = torch.arange(n, device="cuda")
    part = (ids < n // 4).to(torch.int32)
    half = (graph[1].numel() // n + 1) // 2

    def state(flag):
        z = torch.zeros(n, dtype=torch.int32, device="cuda")
        return z.clone(), z, part.clone(), flag.to(torch.int32)

    bnd, gain, target, upd = state(ids >= n - 70)
    torch.cuda.synchronize()
    h.update_vertex_info(graph, 2, part, upd, bnd, gain, target)
    p = part.cpu().numpy()
    for v in range(n - 70, n):
        q = p[_row(graph, v)]
        d = (int((q == 1).sum()) - int((q == 0).sum())) % 2 ** 32   # the rule compares unsigned
        moves = (q == 1).any() and d > 0
        assert int(bnd[v]) == int((q == 1).any()), v
        assert int(gain[v]) % 2 ** 32 == (d if moves else 0), v
        assert int(target[v]) == (1 if moves else 0), v
    assert int(gain[n - 1]) == 1

    p1, (bnd, gain, target, upd) = part.clone(), state(ids >= n - 70)
    pw = torch.bincount(part).to(torch.int32)
    torch.cuda.synchronize()
    rounds, moves = h.refine(graph, 2, n // 4 + 1, 1024, p1, bnd, gain, target, upd, pw)
    assert (rounds, moves) == (1, 1) and pw.tolist() == [n - n // 4 - 1, n // 4 + 1]
    assert int(p1[n - 1]) == 1 and int((p1 != part).sum()) == 1

    edge = (ids >= n - half) | ((ids >= n // 4 - half) & (ids < n // 4 + half)) | (ids < half)
    p1, (_, gain, target, _) = part.clone(), state(edge)
    pw = torch.bincount(part).to(torch.int32)
    bnd = edge.to(torch.int32)
    torch.cuda.synchronize()
    rounds, moves = h.balance(graph, 2, n - n // 4 - 1, 1, p1, bnd, gain, target, pw)
    assert (rounds, moves) == (1, 1) and pw.tolist() == [n - n // 4 - 1, n // 4 + 1]
    # of each run of candidates the first is kept; the one at the quarter has the larger gain
    assert int(p1[n // 4]) == 1 and int((p1 != part).sum()) == 1


def test_contract(graph, h):
    import torch
    n = graph[3].numel()
    cmap = (torch.arange(n, device="cuda") // 2).to(torch.int32)
    torch.cuda.synchronize()
    cx, ca, cw, cv = h.contract(graph, cmap, n // 2)
    assert int(cv.min()) == 2 and int(cv.max()) == 2
    for c in list(range(n // 2 - 6, n // 2)) + [0, n // 4]:
        ids, cnt = np.unique(np.concatenate([_row(graph, 2 * c), _row(graph, 2 * c + 1)]) // 2, return_counts=True)
        cnt, ids = cnt[ids != c], ids[ids != c]
        b, e = int(cx[c]), int(cx[c + 1])
        assert np.array_equal(ca[b:e].cpu().numpy(), ids) and np.array_equal(cw[b:e].cpu().numpy(), cnt), c


def test_initial_partition_rows(graph, h, orc, gen):
    """No vertex weight: growth ends with its seed, which refinement moves back
    out, so the rows of all members are read and little else is done."""
    import torch
    n = graph[3].numel()
    if n > 1 << 16:
        pytest.skip("the 65536 long rows are one sub-problem of this kind")
    zero = torch.zeros_like(graph[3])
    torch.cuda.synchronize()
    p = h.init_partition((graph[0], graph[1], graph[2], zero), 2, trials=1)
    small = gen.grid27(3, 3, 3)
    want = orc.init_partition(gen.Csr(small.xadj, small.adjncy, small.adjwgt, np.zeros(small.n, np.int32)), 2, trials=1)
    assert np.unique(want).size == 1
    assert torch.unique(p).tolist() == np.unique(want).tolist()
