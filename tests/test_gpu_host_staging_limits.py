"""More handles than the process keeps staging buffers for: all give the result
of one handle, at once and one after another, and a closed handle's share goes
to the next."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_seven_handles_at_once(pkg, gen, tmp_path):
    n = 600000
    rng = np.random.default_rng(17)
    s = rng.integers(0, n, 3 * n)
    g = gen.from_edges(n, s, np.clip(s + rng.integers(-9, 10, 3 * n), 0, n - 1))
    path = str(tmp_path / "small.graph")
    gen.write_metis(gen.delaunay(2000, 3), path)
    hs = [pkg.Handle(0) for _ in range(7)]
    for rep in range(2):
        out = [None] * len(hs)

        def run(i):
            part, cut, _ = hs[i].partition(g.xadj, g.adjncy, g.adjwgt, g.vwgt, 6)
            files = [hs[i].read_metis_device(path) for _ in range(2)]
            out[i] = part, cut, [[t.cpu().numpy() for t in f] for f in files]

        ts = [threading.Thread(target=run, args=(i,)) for i in range(len(hs))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        for part, cut, files in out:
            assert cut == out[0][1] and np.array_equal(part, out[0][0])
            for f in files:
                assert all(np.array_equal(a, b) for a, b in zip(f, out[0][2][0]))
        hs[0].close()
        hs[0] = pkg.Handle(0)
    for h in hs:
        h.close()
    # everything was given back: the whole share can be taken, and no more
    import ctypes
    lib = pkg.lib()
    reserve, unreserve = lib._ZN3gkw13stage_reserveEm, lib._ZN3gkw15stage_unreserveEm
    reserve.argtypes, reserve.restype = [ctypes.c_size_t], ctypes.c_bool
    unreserve.argtypes, unreserve.restype = [ctypes.c_size_t], None
    assert reserve(32 << 20)
    unreserve(32 << 20)
