"""GPU tests of the small cells' projector products (csrc/small.cuh): uneven
projector counts (blocks of 32 rows and their remainders), lone and odd bands,
rows short and long enough for clusters, moving ions, against the restatement.

Tolerance: the FP64 parity bar (test_gpu_parity.py); forces 1e-9 Ha/bohr."""
import numpy as np
import pytest

from cpsd_b200 import api, configs, inputs

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,nion,nb,move", [
    (32, 12.0, 1, 1, 0), (32, 12.0, 5, 9, 0), (32, 12.0, 9, 17, 1), (32, 16.0, 13, 32, 0), (48, 20.0, 16, 5, 1),
    (24, 9.0, 6, 7, 1), (64, 16.0, 3, 25, 0)])
def test_projector_products_match_the_restatement(restatement, n, a, nion, nb, move):
    rng = np.random.default_rng(nion)
    pos = []
    while len(pos) < nion:
        p = rng.uniform(-0.5 * a, 0.5 * a, size=3)
        d = np.array([p - q for q in pos]).reshape(-1, 3)
        d -= a * np.round(d / a)
        if not len(d) or np.sqrt((d * d).sum(1)).min() > 1.5:
            pos.append(p)
    spec = inputs.CellSpec(name="proj", unit=a, nfft=n, ecut_ry=30.0, species=[configs.H_S, configs.C_SP],
                           katm=[i % 2 for i in range(nion)], positions=np.array(pos), ne=(nb, 0), seed=nion)
    inp = inputs.build_inputs(spec)
    so = oracle.State(inp)
    restatement.run(inp, 2, so, move)
    cell = api.GpuCell(inp)
    cell.set_state(inp.c2, inp.r2)
    cell.run(2, move)
    st = api.State(inp)
    cell.get_state(st)
    cell.close()
    assert np.abs(st.E - so.E).max() < 1e-8 and abs(st.E[0] - so.E[0]) < 1e-9
    assert np.abs(st.c2 - so.c2).max() < 1e-10
    if move:
        assert np.abs(st.fion[:3 * nion] - so.fion[:3 * nion]).max() < 1e-9
