"""The PCG's A·p where a block marches over several planes (2, 3 and 4; a last block with fewer and with as many) and
where the planes take several tiles, ragged ones among them, along j and along k: with conductivities of a few values
(coded) and of more than 256 (as they are), z in FP32 and in FP64; device against the oracle at the PCG's bar of 1e-7, with
the FP64 preconditioner the solves' iterations within one per step (the FP32 one is the device's own: its line solves
are in FP64, so it may need fewer than the oracle's FP32 transforms along three axes, but not more).  The tiling a case is there for is computed by pcg_create's rule from the
kernel's own constants and asserted."""
import os
import re

import numpy as np
import pytest

import cases
import juliatdgl_b200 as T
from juliatdgl_b200 import gpu
from oracle import pyoracle

pytestmark = pytest.mark.gpu

SRC = os.path.join(os.path.dirname(gpu.__file__), "csrc", "pcg.cu")


def _tiling(gr, sms=148):
    """(planes per block, the last block's planes, tiles along j, along k, the last tile's rows short of a whole one)."""
    src = open(SRC).read()
    threads = int(re.search(r"const int AP_T = (\d+);", src).group(1))
    rows, total = int(re.search(r"const int AP_TJ = (\d+)", src).group(1)), threads // 6 - 2
    assert re.search(r"AP_SUM = AP_T / 6 - 2;", src) and "cols = std::max(1, 2 * nsm / tiles)" in src
    up = lambda a, b: -(-a // b)
    ni, nj, nk = gr.Nx - 1, gr.Ny - 1, gr.Nz - 1
    ntj = up(nj, rows)
    tj = up(nj, ntj)
    ntk = up(nk, max(1, min(total - tj, threads // tj)))
    tk = up(nk, ntk)
    chunk = up(ni, max(1, 2 * sms // (ntj * ntk)))
    return chunk, ni - chunk * (up(ni, chunk) - 1), ntj, ntk, ntj * tj - nj, ntk * tk - nk


@pytest.mark.parametrize("many", [False, True])
@pytest.mark.parametrize("f32", [True, False])
@pytest.mark.parametrize("grid,tiling", [((300, 4, 3), (2, 1, 1, 1, 0, 0)), ((640, 3, 3), (3, 1, 1, 1, 0, 0)),
                                         ((900, 2, 2), (4, 3, 1, 1, 0, 0)), ((160, 8, 50), (2, 1, 1, 2, 0, 1)),
                                         ((56, 24, 44), (2, 1, 2, 3, 1, 1)), ((96, 45, 28), (3, 3, 2, 3, 0, 2))])
def test_pcg_planes_and_tiles(grid, tiling, f32, many):
    gr = T.Grid.make(*grid, dx=0.5, buf=2)
    assert _tiling(gr) == tiling
    md = T.two_band(xi_ratio=4.0, κ=2.0)
    st = T.Stepper.make(md, gr, T.box_masks(gr), σvac=0.01, pcg_tol=1e-10, selffield_bc="slab", pcg_f32=f32)
    if many:   # a conductivity of its own on every link
        rng = np.random.default_rng(3)
        st.D = tuple(np.asfortranarray(d * rng.uniform(0.8, 1.2, d.shape)) for d in st.D)
    s = cases.seeded_state(md, gr, st.masks, 0.03, seed=2, amp=1e-2, base=None)
    HJ = T.selffield(st, 0.1)
    n = 3
    o = pyoracle.OracleStepper(st)
    o.upload(s)
    gs = gpu.GPUStepper(st)
    try:
        a, b = s.copy(), s.copy()
        gs.upload(b)
        assert o.steps(n, 0.03, HJ) == 0 and gs.steps(n, 0.03, HJ) == 0
        o.download(a)
        gs.download(b)
        ia, ib = o.stats().pcg_total_iters, gs.stats().pcg_total_iters
    finally:
        gs.close()
    worst, per = cases.compare_states(b, a)
    assert worst <= 1e-7, per
    assert ia > n and ib - ia <= n and (f32 or ia - ib <= n), (ia, ib)
