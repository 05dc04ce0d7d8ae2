"""A step that fails CalcDT stops before its boundary conditions (step.F90:143-153):
the whole box, ghosts included, is what the update, the ring average and the model
hooks left, bit for bit the CPU restatement's, on grids with rings about the LFM
axis (with and without the Boris correction), with the solar wind and zero-gradient
sides, and in the magnetosphere, where NudgeSW also changes ghost cells across the
E pole (apps/wind.F90:458-484)."""
import numpy as np
import pytest

from mage_b200 import dipole, grids
from mage_b200.gamera import (BACKGROUND_ARRAYS, BC_ION, BC_LFM, BC_PERIODIC, BC_SPHIN, BC_WIND, BC_ZEROGRAD,
                              GAM_EDT_BAD, GamError, GameraGPU, GamParams)
from oracle.oracle import Oracle, OracleParams
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

K = (BC_PERIODIC, BC_PERIODIC)
RINGS = (BC_SPHIN, BC_ZEROGRAD, BC_LFM, BC_LFM) + K
DIPOLE = (BC_SPHIN, BC_WIND, BC_ZEROGRAD, BC_ZEROGRAD) + K
MAGSPHERE = (BC_ION, BC_WIND, BC_LFM, BC_LFM) + K
WIND = dipole.wind_code_units()
BORIS = {"doBoris": True, "Ca": 10.0}
CASES = {
    "rings": ((16, 16, 16), RINGS, (8,), {}),
    "rings-boris": ((16, 16, 16), RINGS, (8,), BORIS),
    "dipole": ((16, 8, 8), DIPOLE, (), {}),
    "magnetosphere": ((16, 8, 16), MAGSPHERE, (8,), {}),
    "magnetosphere-boris": ((16, 8, 16), MAGSPHERE, (8,), BORIS),
}


@pytest.mark.parametrize("case", list(CASES))
def test_whole_box_after_a_failed_step(oracle_built, case):
    N, bc, nch, kw = CASES[case]
    bg = bc[1] == BC_WIND
    xyz = grids.lfm_corners(*N, th0=0.01) if nch else grids.spherical_corners(*N)
    o = Oracle(OracleParams(*N, bc=bc, ringNch=nch, doBackground=bg, M0=dipole.M0 if bg else 0.0,
                            wind=WIND if bg else (0.0,) * 8, **kw), xyz, "gm")
    rng = np.random.default_rng(7)
    ion = (200.0 * rng.standard_normal((3, N[2] + 8, N[1] + 8, 5)),
           200.0 * rng.standard_normal((3, N[2] + 9, N[1] + 9, 6)), dipole.M0, 5.0 / 63.8, True, 2)
    if bc[0] == BC_ION:
        o.set_ionosphere(*ion)
    if bg:
        o.ic_dipole_wind(0.01, 31337)
    else:
        o.ic_blast_wave(x0=6.0, y0=0.7, z0=0.0, rC=3.0, B0=0.3)
    assert o.init_finish() == 0
    assert o.step(2) == 0
    if bc[0] == BC_ION:  # flow back in through the last shell: what NudgeSW turns around
        for g_ in ("Gas", "oGas"):
            o.array(g_)[1][:, 2 + N[1]:, N[0] + 3] = np.abs(o.array(g_)[1][:, 2 + N[1]:, N[0] + 3]) + 1.0
    # limDT0 (step.F90:117-121): dt0 recorded 1e5 times the current dt
    dt0 = 1.0e5 * o.scalars()["dt"]
    o.set_scalars(dt0=dt0)
    g = GameraGPU(GamParams(*N, bc=bc, doBackground=bg, strict=True, dt0=dt0, **kw))
    if nch:
        g.set_rings(nch)
    g.set_geometry(xyz)
    if bg:
        g.set_background({n: o.array(n) for n, _ in BACKGROUND_ARRAYS})
    if bc[0] == BC_ION:
        g.set_ionosphere(*ion)
    if bg:
        g.set_wind(WIND)
    sc = o.scalars()
    g.upload_state(o.array("Gas"), o.array("magFlux"), o.array("Bxyz"), o.array("oGas"), o.array("omagFlux"),
                   sc["time"], sc["otime"], sc["dt"], sc["ts"])
    assert o.step(3) == 1
    with pytest.raises(GamError) as ei:
        g.step_gamera(3)
    assert ei.value.code == GAM_EDT_BAD
    s = g.download_state()
    for k in ("Gas", "magFlux", "Bxyz", "oGas", "omagFlux"):
        assert np.array_equal(s[k], o.array(k)), (k, rel_err(s[k], o.array(k)), int((s[k] != o.array(k)).sum()))
