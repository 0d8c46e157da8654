"""Batches on either side of the rules that a recorded step follows: planes of 49 to 96 rows in row chunks (few planes in
flight) and whole (many), and PCG runs on lines of several nodes a lane (their loops never merge) beside runs that do;
each run with the bits it has alone."""
import numpy as np
import pytest

import cases
import juliatdgl_b200 as T
from juliatdgl_b200 import gpu

pytestmark = pytest.mark.gpu


def _check(runs, steps, contexts):
    """The runs' states after `steps` in a batch are to the bit those of each run alone; `contexts` of them merge."""
    alone = []
    for st, s, H, HJ in runs:
        gs = gpu.GPUStepper(st)
        b = s.copy()
        gs.upload(b)
        gs.steps(steps, H, HJ)
        alone.append(gs.download(b))
        gs.close()
    ctxs = []
    for st, s, H, HJ in runs:
        gs = gpu.GPUStepper(st)
        gs.upload(s.copy())
        ctxs.append(gs)
    bt = gpu.Batch(ctxs)
    try:
        bt.steps(steps, [r[2] for r in runs], [r[3] for r in runs])
        assert bt.one_graph
        assert bt.merge_info["contexts"] == contexts, bt.merge_info
        for gs, (st, s, H, HJ), a in zip(ctxs, runs, alone):
            b = gs.download(s.copy())
            assert np.isfinite(b.G[0]).all() and cases.compare_states(b, a)[0] == 0.0
    finally:
        bt.close()
        for gs in ctxs:
            gs.close()


@pytest.mark.parametrize("rows", [(49, 96), (50, 72), (95, 51)])
def test_two_runs_of_48_to_96_rows(rows):
    runs = [cases.small("rkl_bar", grid=(20 + 13 * q, ny - 1, 4)) for q, ny in enumerate(rows)]
    for r, ny in zip(runs, rows):
        assert r[0].grid.Ny - 1 == ny
    _check(runs, 10, 2)


def test_many_planes_in_flight():
    """More than six planes per SM in all (148 SMs): whole planes, of at most 96 rows and of more."""
    grids = [(240, 52, 4), (230, 63, 5), (250, 95, 3), (220, 40, 4)]
    runs = [cases.small("rkl_bar", grid=g) for g in grids]
    assert sum(r[0].grid.Nx - 1 for r in runs) >= 6 * 148
    _check(runs, 6, 4)


def _pcg(nx, f32):
    gr = T.Grid.make(nx, 8, 4, dx=0.5, buf=2)
    md = T.two_band(xi_ratio=4.0, κ=2.0, gamma_kwt=10.0)
    st = T.Stepper.make(md, gr, T.box_masks(gr), σvac=0.01, pcg_tol=1e-10, pcg_f32=f32)
    return st, T.initial_state(md, gr, st.masks, 0.03), 0.03, T.selffield(st, 0.3)


def test_pcg_runs_on_long_lines():
    runs = [_pcg(64, True), _pcg(150, False), _pcg(230, True)]
    runs += [cases.small("rkl_bar", grid=g) for g in ((90, 8, 4), (40, 10, 5))]
    _check(runs, 10, 2)
