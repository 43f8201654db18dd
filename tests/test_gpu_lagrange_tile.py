"""GPU tests of the tiled Lagrange solver (csrc/kernels.cuh lagrange_tile_kernel)
at the edges of its tiles: 33 to 128 bands, uneven last tiles, two spins,
against the restatement.

Tolerance: the FP64 parity bar (1e-9 Ha, 1e-9 in the Lagrange multipliers,
1e-10 in the coefficients, as test_gpu_parity.py)."""
import itertools

import numpy as np
import pytest

from cpsd_b200 import api, configs, inputs

import oracle

pytestmark = pytest.mark.gpu


def _waves(count):
    g = sorted(itertools.product(range(0, 3), range(-2, 3), range(-2, 3)), key=lambda k: (sum(x * x for x in k), k))
    g = [k for k in g if k > (0, 0, 0)]  # one of each pair +-G
    rows = [(0, 0, 0, 0)] + [k + (l,) for k in g for l in (1, -1)]
    return tuple(rows[:count])


@pytest.mark.parametrize("ne", [(33, 0), (37, 0), (64, 0), (65, 0), (96, 0), (97, 0), (127, 0), (40, 35)])
def test_tiled_solver_matches_the_restatement(restatement, ne):
    spec = configs.small_diamond(24, ne[0], ecut=20.0)
    if ne[1]:
        spec.ispin, spec.ne, spec.start_waves = 2, ne, _waves(ne[0])
    inp = inputs.build_inputs(spec)
    so = oracle.State(inp)
    restatement.run(inp, 2, so)
    cell = api.GpuCell(inp)
    assert cell.tuning()["lagrange_solver"] == 1
    cell.set_state(inp.c2, inp.r2)
    cell.run(2)
    st = api.State(inp)
    cell.get_state(st)
    cell.close()
    assert np.array_equal(np.isnan(st.E), np.isnan(so.E))
    fine = ~np.isnan(so.E)
    assert np.abs(st.E - so.E)[fine].max(initial=0.0) < 1e-8
    fine = ~np.isnan(so.c2)
    assert np.array_equal(fine, ~np.isnan(st.c2))
    assert np.abs(st.c2 - so.c2)[fine].max() < 1e-10
    fine = ~np.isnan(so.lmd)
    assert np.abs(st.lmd - so.lmd)[fine].max(initial=0.0) < 1e-9
