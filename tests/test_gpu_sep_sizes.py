"""The separable inverse at the edges of its transforms' tiles: extents where the components' row chunks differ in number
or kind (48 | 49 and 96 | 97 rows), remainders of the register tiles, the smallest planes, and planes that take the batched products (several planes to a
tile of points, both parities of each extent), lines of one to four nodes a lane and too long for one warp; FP64 and FP32, against
the oracle's dense three-axis transforms at the tolerances of the parity test."""
import numpy as np
import pytest

import juliatdgl_b200 as T
from juliatdgl_b200 import gpu
from juliatdgl_b200.scheme import sep_unknowns
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("nx,ny,nz", [(5, 48, 3), (3, 96, 6), (9, 47, 17), (2, 2, 2), (20, 13, 4), (33, 5, 9),
                                      (3, 64, 64), (2, 63, 70), (6, 100, 55), (2, 140, 49),
                                      (31, 3, 2), (63, 2, 3), (95, 4, 2), (97, 3, 3), (416, 2, 2), (430, 3, 2)])
def test_separable_inverse_sizes(nx, ny, nz, f32):
    gr = T.Grid.make(nx, ny, nz, dx=0.5, buf=1)
    md = T.two_band(xi_ratio=4.0, κ=2.0)
    st = T.Stepper.make(md, gr, T.box_masks(gr), σvac=0.01 if f32 else None, pcg_f32=f32, selffield_bc="slab")
    o = pyoracle.OracleStepper(st)
    gs = gpu.GPUStepper(st)
    try:
        b = np.random.default_rng(5).standard_normal(sep_unknowns(gr))
        ref = o.sep_apply(b, f32=False)
        out = gs.sep_apply(b, f32=f32)
    finally:
        gs.close()
    assert np.max(np.abs(out - ref)) / np.max(np.abs(ref)) <= (2e-6 if f32 else 1e-13)


@pytest.mark.parametrize("a", [0.0, 1e-9, 49.5, 1e4])
@pytest.mark.parametrize("nx,ny,nz", [(2, 2, 2), (3, 5, 4), (33, 6, 9)])
def test_noalloc_closed_factorisation(nx, ny, nz, a):
    """The allocation-free inverse, whose line factorisation is in closed form, against the context's recurrence at the
    same a; the two solves differ by the rounding of pivots of condition 1 + 4a: 1e-15 (1 + 4a), at least 1e-13."""
    import dataclasses

    from test_zz_no_alloc import _noalloc
    gr = T.Grid.make(nx, ny, nz, dx=0.5, buf=1)
    st = T.Stepper.make(T.two_band(xi_ratio=4.0, κ=2.0), gr, T.box_masks(gr), selffield_bc="slab")
    st.fc = dataclasses.replace(st.fc, a=a)
    gs = gpu.GPUStepper(st)
    try:
        b = np.random.default_rng(8).standard_normal(sep_unknowns(gr))
        ref = gs.sep_apply(b)
        out = _noalloc(st, b)
    finally:
        gs.close()
    assert np.max(np.abs(out - ref)) <= max(1e-13, 1e-15 * (1 + 4 * a)) * np.max(np.abs(ref))
