"""GPU tests of the small-cell kernels (csrc/small.cuh: overlaps, Lagrange
fixed point and constraint of at most 32 bands per spin) at the edges of their
8 x 8 tiles, against the restatement.

Tolerance: the FP64 parity bar (1e-9 Ha, 1e-9 in the Lagrange multipliers and
hml, 1e-10 in the coefficients, as test_gpu_parity.py)."""
import numpy as np
import pytest

from cpsd_b200 import api, configs, inputs

import oracle

pytestmark = pytest.mark.gpu

WAVES = [(0, 0, 0, 0)] + [(i, j, k, l) for i, j, k in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0),
                                                       (1, 0, 1), (1, 0, -1), (0, 1, 1), (0, 1, -1))
                          for l in (1, -1)]


@pytest.mark.parametrize("ne", [(1, 0), (2, 0), (7, 0), (8, 0), (9, 0), (16, 0), (17, 0), (24, 0), (25, 0), (32, 0),
                                (9, 8), (17, 3)])
def test_small_cells_match_the_restatement(restatement, ne):
    spec = configs.small_diamond(24, ne[0], ecut=20.0)
    if ne[1]:
        spec.ispin, spec.ne, spec.start_waves = 2, ne, tuple(WAVES[:ne[0]])
    inp = inputs.build_inputs(spec)
    so = oracle.State(inp)
    cell = api.GpuCell(inp)
    cell.set_state(inp.c2, inp.r2)
    for _ in range(2):
        restatement.run(inp, 2, so)
        cell.run(2)
    st = api.State(inp)
    cell.get_state(st)
    ep = cell.epilogue()
    cell.close()
    assert np.array_equal(np.isnan(st.E), np.isnan(so.E))
    fine = ~np.isnan(so.E)
    assert np.abs(st.E - so.E)[fine].max() < 1e-8
    assert np.abs(st.c2 - so.c2).max() < 1e-10
    assert np.abs(st.lmd - so.lmd).max() < 1e-9
    assert np.abs(st.hml - so.hml).max() < 1e-9
    m = ne[0] * ne[0]
    assert np.abs(ep["ortho"][:m].reshape(ne[0], ne[0]) - np.eye(ne[0])).max() < 1e-6
