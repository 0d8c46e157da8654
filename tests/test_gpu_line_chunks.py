"""The separable inverse on lines of every chunk length of the warp-per-line solve (5 to 13 nodes a lane, each with a
full last lane and with a ragged one; its longest line, 416 points, and the first one that takes the staged kernel);
FP64 and FP32, against the oracle's dense three-axis transforms at the tolerances of the parity test."""
import numpy as np
import pytest

import juliatdgl_b200 as T
from juliatdgl_b200 import gpu
from juliatdgl_b200.scheme import sep_unknowns
from oracle import pyoracle

pytestmark = pytest.mark.gpu

# cells along x; a line has one point more
LINES = {5: (129, 159), 6: (160, 191), 7: (200, 223), 8: (230, 255), 9: (260, 287), 10: (300, 319), 11: (330, 351),
         12: (360, 383), 13: (385, 415), 14: (416,)}


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("chunk,nx", [(c, nx) for c, v in LINES.items() for nx in v])
def test_line_chunks(chunk, nx, f32):
    gr = T.Grid.make(nx, 3, 2, dx=0.5, buf=1)
    assert (gr.Nx - 1 + 31) // 32 == chunk
    md = T.two_band(xi_ratio=4.0, κ=2.0)
    st = T.Stepper.make(md, gr, T.box_masks(gr), σvac=0.01 if f32 else None, pcg_f32=f32, selffield_bc="slab")
    o = pyoracle.OracleStepper(st)
    gs = gpu.GPUStepper(st)
    try:
        b = np.random.default_rng(6).standard_normal(sep_unknowns(gr))
        ref = o.sep_apply(b, f32=False)
        out = gs.sep_apply(b, f32=f32)
    finally:
        gs.close()
    assert np.max(np.abs(out - ref)) / np.max(np.abs(ref)) <= (2e-6 if f32 else 1e-13)
