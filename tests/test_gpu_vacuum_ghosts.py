"""A sculpted sample whose vacuum reaches a face of the block while the face's own nodes are no vacuum, and a state that
comes in with Ψ ≠ 0 on the vacuum: the first step's ghosts are formed from what the stages leave there (an RKL/RKC
combination keeps its share), then the vacuum is cleared (neumann!, field.jl:231-246).  Device against the oracle after
the first step and after some more, at the PCG's 1e-7; on the device's own steps twice, to the bit."""
import numpy as np
import pytest

import cases
from juliatdgl_b200 import gpu
from oracle import pyoracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 6])
@pytest.mark.parametrize("kind", ["vac_plain", "vac_kwt", "vac_mat"])
def test_ghosts_beside_vacuum(kind, steps):
    st, s, H, HJ = cases.vacuum(kind)
    gr, vac = st.grid, st.masks.vac
    inside = vac[:, gr.y1].copy()                # the slot's nodes beside the y1 face
    inside[[gr.x1 - 1, gr.x2], :] = False        # (corners of the shell copy two faces)
    assert inside[gr.x1:gr.x2, gr.z1:gr.z2].any()
    vac[:, gr.y1 - 1] = False
    for g in s.G:
        g[vac] = 0.4 + 0.3j
    a = pyoracle.run(st, s, steps, H, HJ)
    ghost = [np.abs(a.G[µ][:, gr.y1 - 1][inside]).max() for µ in range(st.model.N)]
    assert steps > 1 or kind != "vac_kwt" or max(ghost) > 1e-2, ghost   # (an even number of stages: its share stays)
    out = []
    for _ in range(2):
        gs = gpu.GPUStepper(st)
        try:
            b = s.copy()
            gs.upload(b)
            gs.steps(steps, H, HJ)
            out.append(gs.download(b))
        finally:
            gs.close()
    worst, per = cases.compare_states(out[0], a)
    assert worst <= 1e-7, per
    for µ in range(st.model.N):
        assert np.abs(out[0].G[µ][vac]).max() == 0 and np.abs(out[0].F[µ][vac]).max() == 0
        assert np.array_equal(out[0].G[µ], out[1].G[µ]) and np.array_equal(out[0].F[µ], out[1].F[µ])
