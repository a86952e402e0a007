"""Union-find labels, distances and rounds on arbitrary candidate maps against
the oracle: random maps (long cycles), chains in both directions, one big
cycle, mutual pairs, self candidates; sizes around the one-CTA limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random(n, rng):
    return rng.integers(0, n, n)


def _chain_up(n, rng):
    return np.minimum(np.arange(n) + 1, n - 1)


def _chain_down(n, rng):
    return np.maximum(np.arange(n) - 1, 0)


def _cycle(n, rng):
    p = rng.permutation(n)
    c = np.empty(n, np.int64)
    c[p] = np.roll(p, 1)
    return c


def _cycles(n, rng):
    """Cycles of 1 to 7 vertices with trees hanging off them."""
    c = np.arange(n)
    i = 0
    while i < n // 2:
        L = int(rng.integers(1, 8))
        j = min(i + L, n // 2)
        c[i:j] = np.roll(np.arange(i, j), 1)
        i = j
    c[n // 2:] = rng.integers(0, np.maximum(np.arange(n // 2, n), 1))
    p = rng.permutation(n)
    out = np.empty(n, np.int64)
    out[p] = p[c]
    return out


def _pairs(n, rng):
    c = np.arange(n) ^ 1
    return np.where(c < n, c, np.arange(n))


@pytest.mark.parametrize("n", [1, 2, 33, 1000, 16384, 16385, 60000])
@pytest.mark.parametrize("make", [_random, _chain_up, _chain_down, _cycle, _cycles, _pairs])
def test_candidate_maps(handle, orc, n, make):
    import torch
    if n > 2000 and make in (_chain_up, _chain_down, _cycle):
        n = {16384: 2000, 16385: 17000, 60000: 3000}[n]   # the oracle runs one round per hop
    cand = make(n, np.random.default_rng(n)).astype(np.int32)
    root, dist, rounds = handle.union_find(torch.from_numpy(cand).cuda())
    r2, d2, l2 = orc.union_find(cand)
    assert np.array_equal(root.cpu().numpy(), r2)
    assert np.array_equal(dist.cpu().numpy(), d2)
    assert rounds == l2
