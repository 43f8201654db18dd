"""GPU tests of the two-band passes (csrc/pair.cuh) where they can go wrong:
odd band counts and lone bands, spins that never share a pair, spheres at the
edge of the pruned builds (kx, |ky| < 16 at 64, < 24 at 128), spheres too wide
for two bands at 128 FP64, and masks whose lines are not two runs.

Tolerance: the FP64 parity bar (1e-9 Ha, 1e-10 in the coefficients, as
test_gpu_parity.py); FP32 transforms keep the energy within 1e-6 relative of
FP64 per step (test_mixed_precision_tracks_fp64's bar).
"""
import dataclasses

import numpy as np
import pytest

from cpsd_b200 import api, configs, inputs, lib

import oracle

pytestmark = pytest.mark.gpu


def _cell(n, a, ecut, ne, holes=0):
    pos = configs.diamond_positions(a, 1, 0.05, 3)
    spec = inputs.CellSpec(name="pair", unit=a, nfft=n, ecut_ry=ecut, species=[configs.C_SP], katm=[0] * 8,
                           positions=pos, ne=ne, ispin=2 if ne[1] else 1, seed=5)
    if ne[1]:
        # near-uniform densities: the reference's spin-polarised exchange is NaN elsewhere
        spec.start_waves = ((0, 0, 0, 0), (1, 0, 0, 1), (1, 0, 0, -1), (0, 1, 0, 1), (0, 1, 0, -1))[:ne[0]]
    if not holes:
        return inputs.build_inputs(spec)
    inp = inputs.build_inputs(dataclasses.replace(spec, ne=(1, 0)))
    # drop whole columns (kx, ky) with their mirror on kx = 0: the lines are no longer two runs
    rng = np.random.default_rng(9)
    nh = n // 2 + 1
    m = inp.masker1.reshape(n, n, nh).copy()
    for _ in range(holes):
        i, j = int(rng.integers(0, 4)), int(rng.integers(1, 4))
        m[:, j, i] = 0
        if i == 0:
            m[:, (n - j) % n, i] = 0
    m = m.reshape(-1)
    return dataclasses.replace(inp, ne=np.array(ne, dtype=np.int32), masker1=m, masker=np.repeat(m, 2).astype(np.int32),
                               tg=inp.tg * m, vc=inp.vc * m, vg=inp.vg * m,
                               c2=inputs.random_orbitals(n, m, ne[0], 5).reshape(-1))


def _run(inp, precision=lib.CPSD_PREC_FP64, **tuning):
    cell = api.GpuCell(inp, precision=precision)
    cell.set_state(inp.c2, inp.r2)
    if tuning:
        cell.set_tuning(**tuning)
    cell.run(2)
    st = api.State(inp)
    cell.get_state(st)
    cell.close()
    return st


CELLS = {
    "16_one_band": (16, 6.0, 12.0, (1, 0)),
    "24_odd": (24, 9.0, 20.0, (3, 0)),
    "24_spin": (24, 10.26, 20.0, (5, 4)),
    "32_wide": (32, 16.0, 30.0, (5, 0)),
    "48_wide": (48, 24.0, 30.0, (2, 0)),
    "64_pruned_edge": (64, 15.4, 40.0, (3, 0)),
    "64_past_edge": (64, 16.4, 40.0, (2, 0)),
    "64_spin": (64, 10.26, 40.0, (3, 2)),
    "128_pruned": (128, 20.5, 40.0, (3, 0)),
    "128_past_edge": (128, 25.0, 40.0, (2, 0)),
    "128_one_band_pass": (128, 34.0, 40.0, (2, 0)),
}


@pytest.mark.parametrize("name", list(CELLS))
def test_pairs_match_the_restatement(restatement, name):
    n, a, ecut, ne = CELLS[name]
    inp = _cell(n, a, ecut, ne)
    so = oracle.State(inp)
    restatement.run(inp, 2, so)
    st = _run(inp)
    assert np.abs(st.E - so.E).max() < 1e-8 and abs(st.E[0] - so.E[0]) < 1e-9
    assert np.abs(st.c2 - so.c2).max() < 1e-10
    assert np.abs(st.dn - so.dn).max() < 1e-11
    if not ne[1]:
        sm = _run(inp, lib.CPSD_PREC_MIXED)
        assert abs(sm.E[0] - so.E[0]) < 2e-6 * abs(so.E[0])


def test_lines_that_are_not_two_runs(restatement):
    inp = _cell(32, 12.0, 30.0, (3, 0), holes=4)
    so = oracle.State(inp)
    restatement.run(inp, 2, so)
    st = _run(inp)
    assert abs(st.E[0] - so.E[0]) < 1e-9
    assert np.abs(st.c2 - so.c2).max() < 1e-10


@pytest.mark.parametrize("chunks", [1, 2, 4])
def test_chunks_of_odd_sizes(restatement, chunks):
    """Density chunks with lone bands inside, one pair or several per CTA."""
    inp = _cell(32, 12.0, 25.0, (7, 0))
    so = oracle.State(inp)
    restatement.run(inp, 2, so)
    st = _run(inp, density_chunks=chunks)
    assert abs(st.E[0] - so.E[0]) < 1e-9
    assert np.abs(st.dn - so.dn).max() < 1e-11
