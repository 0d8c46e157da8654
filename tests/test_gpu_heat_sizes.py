"""The heat model's sweep by planes at its edges: fewer columns than a warp, more than a block's threads, more than its
shared memory holds, spacings whose squares are powers of two and not, two cells along each axis; device against the
oracle, Ψ and links at the exact-solve tolerance 1e-11, the temperature field too."""
import numpy as np
import pytest

import cases
import juliatdgl_b200 as T
from juliatdgl_b200 import abi, gpu
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,dx,steps", [((2, 2, 2), 0.5, 12), ((9, 5, 4), 0.4, 12), ((4, 40, 30), 0.5, 6),
                                           ((4, 40, 30), 0.3, 6), ((3, 130, 110), 0.5, 2)])
def test_heat_sweep_sizes(grid, dx, steps):
    gr = T.Grid.make(*grid, dx=dx)
    md = T.two_band(xi_ratio=4.0, κ=2.0, gamma_kwt=3.0)
    mk = T.box_masks(gr)
    st = T.Stepper.make(md, gr, mk, selffield_bc="slab", heat=T.Heat(eta=0.5, joule=True))
    s = T.initial_state(md, gr, mk, 0.03)
    HJ = T.selffield(st, 0.3)
    o = pyoracle.OracleStepper(st)
    o.upload(s)
    gs = gpu.GPUStepper(st)
    try:
        a, b = s.copy(), s.copy()
        gs.upload(b)
        o.steps(steps, 0.03, HJ)
        gs.steps(steps, 0.03, HJ)
        o.download(a)
        gs.download(b)
        ca, cb = abi.Carry(st), abi.Carry(st)
        o.get_carry(ca)
        gs.get_carry(cb)
    finally:
        gs.close()
    worst, per = cases.compare_states(b, a)
    assert worst <= 1e-11, per
    d = np.max(np.abs(cb.heat_theta - ca.heat_theta))
    assert np.max(np.abs(ca.heat_theta)) > 0 and d <= 1e-11 * np.max(np.abs(ca.heat_theta)), d
