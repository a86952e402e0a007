"""Host arrays above and below the staged-copy limit, pageable and pinned, give
the same partition as device arrays (the copies are exact); several handles
copy at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pin(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.int32, pin_memory=True)
    t.copy_(torch.from_numpy(a))
    return t.numpy()


@pytest.mark.parametrize("n", [100000, 530000, 700000])   # 2.4, 12.7 and 16.8 MB of neighbour ids
def test_host_copies(handle, gen, n):
    import torch
    rng = np.random.default_rng(n)
    s = rng.integers(0, n, 3 * n)
    g = gen.from_edges(n, s, np.clip(s + rng.integers(-30, 31, 3 * n), 0, n - 1), rng.integers(1, 5, 3 * n))
    host = [g.xadj, g.adjncy, g.adjwgt, g.vwgt]
    dev = [torch.from_numpy(a).cuda() for a in host]
    part = torch.empty(n, dtype=torch.int32, device="cuda")
    cut, _ = handle.partition_device(*dev, 4, part)
    want = part.cpu().numpy()
    for arrays in (host, [_pin(a) for a in host]):
        got, c, _ = handle.partition(*arrays, 4)
        assert c == cut and np.array_equal(got, want)
    parts, cuts = handle.partition_multi_k(*host, [2, 4, 8, 4, 2, 3, 5])
    assert cuts[1] == cut and np.array_equal(parts[1], want) and np.array_equal(parts[3], want)


def test_host_copies_from_two_handles(pkg, gen):
    n = 600000
    rng = np.random.default_rng(5)
    s = rng.integers(0, n, 3 * n)
    g = gen.from_edges(n, s, np.clip(s + rng.integers(-9, 10, 3 * n), 0, n - 1))
    out = [None, None]

    def run(i):
        h = pkg.Handle(0)
        for _ in range(3):
            out[i] = h.partition(g.xadj, g.adjncy, g.adjwgt, g.vwgt, 6)[:2]
        h.close()

    t = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert out[0][1] == out[1][1] and np.array_equal(out[0][0], out[1][0])
