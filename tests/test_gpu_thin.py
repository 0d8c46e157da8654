"""Blocks of two and three cells along an axis, where every node of a band stage has ghosts beside it (the stages form an
intermediate stage's ghosts, the faces of the frame rate and the rotated links themselves), device against the oracle
at the tolerance of the exact-solve cases; F outside the block comes in nonzero (the reference's copy of a stage buffer
clears it, its in-place stages keep it)."""
import numpy as np
import pytest

import cases
from juliatdgl_b200 import gpu
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(2, 5, 3), (9, 2, 2), (3, 4, 2)])
@pytest.mark.parametrize("kind,kw", [("rkl_bar", {}), ("rkc_kwt_rotframe", {}), ("kwt_substeps_rotframe", {}),
                                     ("euler_substeps", {}), ("rkc_kwt_rotframe", dict(noise=1e-3, noise_seed=5)),
                                     ("drag_substeps", {})])
def test_thin_blocks(kind, kw, grid):
    st, s, H, HJ = cases.small(kind, grid=grid, **kw)
    s = pyoracle.run(st, s, 5, H, HJ)
    gr = st.grid
    out = np.ones(gr.node, dtype=bool)
    out[gr.x1 - 1:gr.x2 + 1, gr.y1 - 1:gr.y2 + 1, gr.z1 - 1:gr.z2 + 1] = False
    for f in s.F:
        f[out] = 0.25
    a = pyoracle.run(st, s, 12, H, HJ)
    gs = gpu.GPUStepper(st)
    try:
        b = s.copy()
        gs.upload(b)
        gs.steps(12, H, HJ)
        gs.download(b)
    finally:
        gs.close()
    worst, per = cases.compare_states(b, a)
    assert worst <= (1e-10 if kw else 1e-11), per
