"""The heat model on blocks whose cross-section is much larger than their length (the sweep has far more planes than a
column has nodes, so that each plane's slot is taken again many times): its device memory is the field and two arrays of
the block at most, with the last two planes of a cross-section too large for shared memory, and the device matches the
oracle at the exact-solve tolerance 1e-11, the temperature field too."""
import numpy as np
import pytest

import cases
import juliatdgl_b200 as T
from juliatdgl_b200 import abi, gpu
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _stepper(grid, heat):
    gr = T.Grid.make(*grid, dx=0.4)
    md = T.two_band(xi_ratio=4.0, κ=2.0, gamma_kwt=3.0)
    mk = T.box_masks(gr)
    kw = dict(heat=T.Heat(eta=0.5, joule=True)) if heat else {}
    return md, T.Stepper.make(md, gr, mk, selffield_bc="slab", **kw)


@pytest.mark.parametrize("grid", [(2, 60, 44), (3, 33, 70), (3, 130, 110), (90, 4, 3)])
def test_heat_memory_is_the_blocks(grid):
    used = []
    for heat in (False, True):
        gs = gpu.GPUStepper(_stepper(grid, heat)[1])
        used.append(gs.device_bytes)
        gs.close()
    gr = T.Grid.make(*grid, dx=0.4)
    field = 8 * (gr.Nx + 1) * (gr.Ny + 1) * (gr.Nz + 1)
    cross = (gr.y2 - gr.y1) * (gr.z2 - gr.z1)
    prev = 16 * cross if 16 * cross > 200 * 1024 else 0
    assert used[1] - used[0] <= 3 * field + prev + 4 * 512, (used, field, prev)


@pytest.mark.parametrize("grid,steps", [((2, 60, 44), 6), ((3, 33, 70), 6), ((90, 4, 3), 12)])
def test_heat_sweep_of_reused_slots(grid, steps):
    md, st = _stepper(grid, True)
    s = T.initial_state(md, st.grid, st.masks, 0.03)
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
