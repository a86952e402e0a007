"""Handle.set_tuning changes the shapes it names and no others (no device
needed: the library's table is stood in for)."""
import ctypes

import pytest


class Table:
    """gkw_get_tuning and gkw_set_tuning over one table."""

    def __init__(self, pkg):
        self.t = pkg.Tuning((ctypes.c_int32 * 4)(2, 8, 16, 32), 128, 16, 80000, 512)

    def gkw_get_tuning(self, h, out):
        ctypes.memmove(out, ctypes.byref(self.t), ctypes.sizeof(self.t))
        return 0

    def gkw_set_tuning(self, h, t):
        ctypes.memmove(ctypes.byref(self.t), t, ctypes.sizeof(self.t))
        return 0


@pytest.mark.parametrize("named", [
    {}, {"match_lanes": (4, 4, 8, 16)}, {"level_verts_per_cta": 1024}, {"level_min_ctas": 64},
    {"coarsen_fused_max_n": 0}, {"coarsen_verts_per_cta": 256}, {"level_verts_per_cta": 64, "level_min_ctas": 1}])
def test_only_the_named_shapes_change(pkg, monkeypatch, named):
    table = Table(pkg)
    monkeypatch.setattr(pkg, "lib", lambda: table)
    h = pkg.Handle.__new__(pkg.Handle)
    h._h = None
    want = table.t.as_dict()
    h.set_tuning(**named)
    want.update({k: list(v) if k == "match_lanes" else v for k, v in named.items()})
    assert table.t.as_dict() == want
