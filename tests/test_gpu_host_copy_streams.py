"""Pageable arrays above the staged-copy limit on streams a caller may name: a
created stream, the legacy default stream and the per-thread default stream,
which is another stream on every host thread and so cannot be shared by the
threads of a staged copy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEGACY, PER_THREAD = 1, 2   # cudaStreamLegacy, cudaStreamPerThread


@pytest.mark.parametrize("stream", ["created", "null", "legacy", "per_thread"])
def test_staged_copies_on_a_callers_stream(pkg, gen, stream):
    import torch
    n = 2200000   # 8.8 MB of vertex arrays and part ids, 35 MB and more of entries
    rng = np.random.default_rng(8)
    s = rng.integers(0, n, 2 * n)
    g = gen.from_edges(n, s, np.clip(s + rng.integers(-20, 21, 2 * n), 0, n - 1), rng.integers(1, 5, 2 * n))
    arrays = (g.xadj, g.adjncy, g.adjwgt, g.vwgt)
    own = pkg.Handle(0)
    want, wcut, _ = own.partition(*arrays, 4)
    own.close()
    keep = torch.cuda.Stream()
    h = pkg.Handle(0)
    h.set_stream({"created": keep.cuda_stream, "null": 0, "legacy": LEGACY, "per_thread": PER_THREAD}[stream])
    for _ in range(2):
        part, cut, _ = h.partition(*arrays, 4)
        assert cut == wcut and np.array_equal(part, want)
    parts, cuts = h.partition_multi_k(*arrays, [4, 2])
    assert cuts[0] == wcut and np.array_equal(parts[0], want)
    h.close()
