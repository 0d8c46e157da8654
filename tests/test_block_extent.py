"""The host-side parameter check refuses a block one cell thick along an axis (no inner node: the heat model's sweep
would place its faces before its arrays, the band stages would launch no block) and takes two cells."""
import ctypes as C

import pytest

import cases
from juliatdgl_b200 import abi, gpu


def _supported(p):
    buf = C.create_string_buffer(256)
    return gpu.lib().tdgl_supported(C.byref(p), buf, 256), buf.value.decode()


@pytest.mark.parametrize("axis", "xyz")
@pytest.mark.parametrize("kind", ["rkl_bar", "heat_joule"])
def test_one_cell_is_refused(kind, axis):
    st, s, H, HJ = cases.small(kind)
    p, keep = abi.pack_params(st)
    lo = getattr(p.grid, axis + "1")
    setattr(p.grid, axis + "2", lo + 1)          # two cells: nodes lo, lo + 1 (inner) and lo + 2
    ok, why = _supported(p)
    assert ok, why
    for hi in (lo, lo - 1):                      # one cell, none
        setattr(p.grid, axis + "2", hi)
        ok, why = _supported(p)
        assert not ok and "two cells" in why, (hi, why)
