"""The conductivities' byte codes of the PCG's A·p: a context whose links have at most 256 values keeps a byte per link
and component, one with more keeps none of it (the arrays are allocated once the values are known to be few)."""
import numpy as np
import pytest

import juliatdgl_b200 as T
from juliatdgl_b200 import gpu

pytestmark = pytest.mark.gpu


def _bytes(values):
    """Device memory of a 24×12×8-cell context whose inner links hold `values` conductivities."""
    gr = T.Grid.make(24, 12, 8, dx=0.5, buf=2)
    st = T.Stepper.make(T.two_band(xi_ratio=4.0, κ=2.0), gr, T.box_masks(gr), σvac=0.01, selffield_bc="slab")
    each = []
    for q, d in enumerate(st.D):
        v = 0.5 + (np.arange(d.size) % values) / 1024 if q == 0 else np.full(d.size, 0.5)
        each.append(np.asfortranarray(v.reshape(d.shape, order="F")))
    st.D = tuple(each)
    gs = gpu.GPUStepper(st)
    try:
        return gs.device_bytes, (gr.Nx + 1) * (gr.Ny + 1) * (gr.Nz + 1)
    finally:
        gs.close()


def test_codes_only_where_they_serve():
    few, n = _bytes(200)          # 201 values with the zeros outside the ranges
    full, _ = _bytes(255)         # 256 with them
    many, _ = _bytes(600)
    assert few == full and 3 * n <= few - many <= 3 * n + 3 * 16, (few, full, many, n)
