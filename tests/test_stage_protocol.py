"""The projection's staged appends (ph_project, csrc/refine.cu) under random
schedules of a CTA's warps, as a CPU model.

Each chunk, every warp appends its boundary vertices to the stage and passes the
block barrier; then all warps must decide alike whether to flush, since the
flush has barriers of its own.  A decision that reads the stage's shared count
is not uniform: a warp that is ahead may have appended entries of the next chunk
by then.  The count summed at the barriers is the same in every warp."""
import random

import pytest

WARPS, LANES, STAGE = 4, 8, 64


def _run(rng, chunks, by_barrier):
    """Warps step in random order; returns the appended entries, or None when
    warps of one CTA wait at different barriers or the stage overflows."""
    cta = WARPS * LANES
    out, stage, cnt = [], [], [0]
    arrived, counted = {}, [0]

    def warp(w):
        have = 0
        for c in range(len(chunks)):
            mine = chunks[c][w]
            if c and mine:
                yield "run"               # loads of the chunk: other warps run meanwhile
            if cnt[0] + mine > STAGE:
                yield "overflow"
            stage.extend((c, w, i) for i in range(mine))
            cnt[0] += mine
            total = yield ("barrier", "chunk", mine)
            have += total
            yield "run"
            if (have if by_barrier else cnt[0]) > STAGE - cta:
                if w == 0:
                    out.extend(stage)
                yield ("barrier", "base", 0)
                yield ("barrier", "copied", 0)
                if w == 0:
                    stage.clear()
                    cnt[0] = 0
                yield ("barrier", "cleared", 0)
                have = 0
        yield ("barrier", "end", 0)
        if w == 0:
            out.extend(stage)

    ws = {w: warp(w) for w in range(WARPS)}
    send = dict.fromkeys(ws)
    while ws:
        ready = [w for w in ws if w not in arrived]
        if not ready:
            if len({a[1] for a in arrived.values()}) != 1:
                return None               # some flush, some do not
            total = sum(a[2] for a in arrived.values())
            for w in arrived:
                send[w] = total
            arrived.clear()
            continue
        w = rng.choice(ready)
        try:
            step = ws[w].send(send[w])
        except StopIteration:
            del ws[w]
            continue
        send[w] = None
        if step == "overflow":
            return None
        if step != "run":
            arrived[w] = step
    return out


def _chunks(rng, n, dense):
    return [[rng.randint(LANES // 2, LANES) if rng.random() < dense else rng.randint(0, 2) for _ in range(WARPS)]
            for _ in range(n)]


@pytest.mark.parametrize("dense", [0.2, 0.6, 1.0])
def test_count_of_the_barriers(dense):
    rng = random.Random(int(dense * 10))
    for _ in range(400):
        chunks = _chunks(rng, 12, dense)
        out = _run(rng, chunks, True)
        want = sorted((c, w, i) for c, row in enumerate(chunks) for w, m in enumerate(row) for i in range(m))
        assert out is not None and sorted(out) == want


def test_shared_count_would_split_the_cta():
    rng = random.Random(1)
    assert any(_run(rng, _chunks(rng, 12, 0.6), False) is None for _ in range(400))
