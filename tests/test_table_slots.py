"""The hash tables' size for coarse rows of any accepted length (no device needed;
the function is the library's own, called by its C++ name in a process that is
given up on if it does not end)."""
import ctypes
import os
import subprocess
import sys

ROWS = [0, 1, 31, 32, 33, 64, 65, 4096, 4097, (1 << 29) + 1, (1 << 30) - 1, 1 << 30, (1 << 30) + 1, (1 << 31) - 2,
        (1 << 31) - 1]


def check():
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import __graft_entry__ as ge
    slots = ge.load_package().lib()._ZN3gkw11table_slotsEj
    slots.argtypes, slots.restype = [ctypes.c_uint32], ctypes.c_uint32
    for n in ROWS:
        s = slots(n)
        assert s & (s - 1) == 0 and s >= 64, n
        assert s == (1 << 31) if n > 1 << 30 else 2 * n <= s < max(4 * n, 128), n


def test_every_row_length_ends():
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]


if __name__ == "__main__":
    check()
