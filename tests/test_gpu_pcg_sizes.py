"""The PCG's A·p at the edges of its tiles along j (24 | 25 rows and more, a block of two cells along each axis; one plane
per block and one tile along k), with conductivities of a few values (coded) and of more than 256 (as they are), each
preconditioner; device against the oracle at the PCG's bar of 1e-7, the solves' iterations within one per step."""
import numpy as np
import pytest

import cases
import juliatdgl_b200 as T
from juliatdgl_b200 import gpu
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("grid,pcg", [((4, 21, 10), dict()), ((5, 22, 11), dict()), ((2, 2, 2), dict()),
                                      ((40, 3, 2), dict(pcg_f32=False)), ((3, 45, 3), dict(pcg_f32=False, pcg_fast=False))])
def test_pcg_tile_edges(grid, pcg, many):
    gr = T.Grid.make(*grid, dx=0.5, buf=2)
    md = T.two_band(xi_ratio=4.0, κ=2.0)
    st = T.Stepper.make(md, gr, T.box_masks(gr), σvac=0.01, pcg_tol=1e-10, selffield_bc="slab", **pcg)
    if many:   # a conductivity of its own on every link
        rng = np.random.default_rng(3)
        st.D = tuple(np.asfortranarray(d * rng.uniform(0.8, 1.2, d.shape)) for d in st.D)
    s = cases.seeded_state(md, gr, st.masks, 0.03, seed=2, amp=1e-2, base=None)
    HJ = T.selffield(st, 0.1)
    o = pyoracle.OracleStepper(st)
    o.upload(s)
    gs = gpu.GPUStepper(st)
    try:
        a, b = s.copy(), s.copy()
        gs.upload(b)
        n = 8
        assert o.steps(n, 0.03, HJ) == 0 and gs.steps(n, 0.03, HJ) == 0
        o.download(a)
        gs.download(b)
        ia, ib = o.stats().pcg_total_iters, gs.stats().pcg_total_iters
    finally:
        gs.close()
    worst, per = cases.compare_states(b, a)
    assert worst <= 1e-7, per
    assert ia > n and abs(ia - ib) <= n, (ia, ib)
