"""gkw_predict_footprint covers what the pipeline allocates on graphs with fewer
entries than vertices, whose components stay on every level (no device needed).

The allocations are restated here from their sizes in bytes: per vertex and
entry of a level in the hierarchy (coarsen_level), of the refinement context
(refine_create), of a large level's coarsening scratch (run_large_level) and of
the initial partition's (device_init_partition_body)."""
import math

import pytest


def hierarchy(levels, n, m):
    up = 4 * (n + 1) + 8 * m + 4 * n + 4 * n                       # the input and the part ids
    return up + sum(12 * a + 4 + 8 * b for a, b in levels)         # cmap, cxadj, cvwgt and rows at upper bounds


def refinement(n):
    # part and boundary twice, gain, target; updflag, inP, U, P twice, msrc, cw, btarget, bgain, blist, bmark; cands, cinfo
    return 4 * 6 * n + 4 * 11 * n + 8 * 2 * n


def coarsening(a, b, cap=6):
    base = 8 * a + 4 * a + 4 * cap * a                             # sums, mcnt, memtab
    groups = 16 * a + 8 * a + 4 * a + 8 * a + 4 * a + 4 * a + 4 * a   # union-find block, keys, gsize, grec, goff, members, list
    rows = 5 * 4 * a + 8 * b                                       # rowlen, cnt, ub, heavy, mid; sadj and swgt
    return base + max(groups, rows)


def initial(a, b, k):
    state = 8 * 2 * 4 * a + 8 * 8 * a + 8 * 8 * (a // 32 + k + 2) + 8 * 8 * (a // 1024 + k + 2)
    large = 16 * a + 8 * b + 8 * a + 8 * 2 * 4 * a                 # headers, rows, sides, growth words
    return 3 * 4 * a + 8 * k + state + large + 16 * k


def needed(levels, n, m, k):
    scratch = max([coarsening(a, b) for a, b in levels] + [initial(*levels[-1], k)])
    return hierarchy(levels, n, m) + refinement(n) + scratch


def edgeless(n):
    return 0, [(n, 0)]


def matching(n):
    return n // 2 * 2, [(n, n // 2 * 2), (n - n // 2, 0)]


def mesh_among_isolated(n, share):
    a = int(n * share)
    m, levels = 6 * a, [(n, 6 * a)]
    while a > 50:
        a = int(a * 0.35)
        levels.append((n - int(n * share) + a, 6 * a))
    return m, levels


@pytest.mark.parametrize("n", [200_000, 3_000_000, 100_000_000])
@pytest.mark.parametrize("k", [2, 64, 1000])
def test_components_that_stay(pkg, n, k):
    cases = {"edgeless": edgeless(n), "matching": matching(n)}
    cases.update({f"mesh_{s}": mesh_among_isolated(n, s) for s in (0.001, 0.01, 0.05, 0.1, 0.15)})
    for name, (m, levels) in cases.items():
        assert m <= n
        assert pkg.predict_footprint(n, m, k) >= needed(levels, n, m, k), name


def test_ordinary_graphs_as_before(pkg):
    """From 1.5 entries a vertex on, and an initial partition far smaller than
    the graph, the coarsening's scratch decides and the prediction is the sum it was."""
    for n, m, k in ((1 << 20, 6291384, 64), (12_000_000, 27_000_000, 256), (4_000_000, 24_000_000, 256),
                    (960_000, 24_000_000, 64)):
        want = 4 * (n + 1) + 8 * m + 8 * n + 1.5 * (12 * n + 8 * m) + 10 * n + 96 * n + 32 * k + 64 * n + 24 * m
        assert math.isclose(pkg.predict_footprint(n, m, k), want + (16 << 20), rel_tol=1e-9)
