"""The process-wide limits of the host staging: bytes of kept buffers and helper
threads are handed out up to a total and come back (no device needed).  The
functions are the library's own, called by their C++ names, in a process of
their own: other handles hold shares of this one's."""
import ctypes
import os
import subprocess
import sys
import threading

import pytest

BUFFER = 32 << 20   # what one handle keeps for its copies


def staging():
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import __graft_entry__ as ge
    lib = ge.load_package().lib()
    reserve, unreserve = lib._ZN3gkw13stage_reserveEm, lib._ZN3gkw15stage_unreserveEm
    take, give = lib._ZN3gkw18stage_take_helpersEi, lib._ZN3gkw20stage_return_helpersEi
    reserve.argtypes, reserve.restype = [ctypes.c_size_t], ctypes.c_bool
    unreserve.argtypes, unreserve.restype = [ctypes.c_size_t], None
    take.argtypes, take.restype = [ctypes.c_int], ctypes.c_int
    give.argtypes, give.restype = [ctypes.c_int], None
    return reserve, unreserve, take, give


def bytes_of_256_handles():
    reserve, unreserve, _, _ = staging()
    got = [reserve(BUFFER) for _ in range(256)]
    assert sum(got) == 4
    assert not reserve(1)
    unreserve(BUFFER)
    assert reserve(BUFFER // 2) and reserve(BUFFER // 2) and not reserve(1)
    for _ in range(4):
        unreserve(BUFFER)
    assert reserve(4 * BUFFER) and not reserve(1)
    unreserve(4 * BUFFER)
    assert not reserve(4 * BUFFER + 1)


def helpers_of_256_copies():
    _, _, take, give = staging()
    got = [take(7) for _ in range(256)]
    assert 0 <= sum(got) <= 28 and all(0 <= x <= 7 for x in got)
    assert take(7) == 0
    for x in got:
        if x:
            give(x)
    assert [take(7) for _ in range(256)] == got


def concurrent_copies_return_what_they_take():
    _, _, take, give = staging()
    first = take(28)
    give(first)
    most, held, lock = [0], [0], threading.Lock()

    def copies():
        for _ in range(300):
            n = take(7)
            with lock:
                held[0] += n
                most[0] = max(most[0], held[0])
            with lock:
                held[0] -= n
            if n:
                give(n)

    ts = [threading.Thread(target=copies) for _ in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert most[0] <= 28 and take(28) == first


CHECKS = [bytes_of_256_handles, helpers_of_256_copies, concurrent_copies_return_what_they_take]


@pytest.mark.parametrize("check", [c.__name__ for c in CHECKS])
def test_limits(check):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), check], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


if __name__ == "__main__":
    {c.__name__: c for c in CHECKS}[sys.argv[1]]()
