"""The update leaves out the ghosts that the step's periodic boundaries fill: the
whole box, ghosts included, equals the CPU restatement bit for bit after steps,
and after a step that failed CalcDT, which stops before its boundaries with the
ghosts of its start (step.F90:143-153). With AB3 the fluxes of every face move
on; in 2.5-D the slabs of k are not shrunk."""
import numpy as np
import pytest

from mage_b200.gamera import GAM_EDT_BAD, GamError
from tests.helpers import gpu_from_oracle, make_oracle

pytestmark = pytest.mark.gpu

SIZES = [(16, 4, 4), (24, 9, 12), (40, 17, 1)]


@pytest.mark.parametrize("fail", [False, True], ids=["steps", "failed"])
@pytest.mark.parametrize("ab3", [False, True], ids=["ab2", "ab3"])
@pytest.mark.parametrize("N", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
def test_whole_box_matches_oracle(oracle_built, N, ab3, fail):
    o, _ = make_oracle("ot" if N[2] == 1 else "bw", N, variant="gm", doAB3=ab3)
    assert o.step(2) == 0
    kw = {"doAB3": ab3}
    if fail:  # limDT0 (step.F90:117-121): dt0 recorded 1e5 times the current dt
        kw["dt0"] = 1.0e5 * o.scalars()["dt"]
        o.set_scalars(dt0=kw["dt0"])
    g = gpu_from_oracle(o, strict=True, **kw)
    if ab3:
        g.set_oostate(o.array("oomagFlux"), o.scalars()["ootime"])
    assert o.step(3) == (1 if fail else 0)
    if fail:
        with pytest.raises(GamError) as ei:
            g.step_gamera(3)
        assert ei.value.code == GAM_EDT_BAD
    else:
        g.step_gamera(3)
    s = g.download_state()
    for k in ("Gas", "magFlux", "Bxyz"):
        assert np.array_equal(s[k], o.array(k)), k


@pytest.mark.parametrize("ab3", [False, True], ids=["ab2", "ab3"])
@pytest.mark.parametrize("N", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
def test_slots_past_the_last_cell(oracle_built, N, ab3):
    """magFlux has a layer past the last cell across each component's direction that
    no face is in: what State has there stays, whatever oState has."""
    o, _ = make_oracle("ot" if N[2] == 1 else "bw", N, variant="gm", doAB3=ab3)
    for n, name in enumerate(("magFlux", "omagFlux")):
        for d in range(3):
            for a in range(3):
                if a != d:
                    sl = [slice(None)] * 3
                    sl[2 - a] = -1
                    o.array(name)[d][tuple(sl)] = 1.0 + n + 0.1 * d + 0.01 * a
    g = gpu_from_oracle(o, strict=True, doAB3=ab3)
    if ab3:
        g.set_oostate(o.array("oomagFlux"), o.scalars()["ootime"])
    for n in (1, 2):
        assert o.step(n) == 0
        g.step_gamera(n)
        s = g.download_state()
        for k in ("Gas", "magFlux", "Bxyz"):
            assert np.array_equal(s[k], o.array(k)), (n, k)
        if ab3:
            assert np.array_equal(g.get_oostate()["oomagFlux"], o.array("oomagFlux")), n


def test_no_steps_change_nothing(oracle_built):
    """A call for no steps leaves the times alone, also where a step would first move
    oState's time one dt back (mhdgroup.F90:25-31)."""
    o, _ = make_oracle("ot", (16, 4, 4), variant="gm")
    g = gpu_from_oracle(o, strict=True)
    gas, mf, dt = o.array("Gas"), o.array("magFlux"), o.scalars()["dt"]
    g.upload_state(gas, mf, o.array("Bxyz"), gas, mf, 1.0, 1.0, dt, 5)
    g.step_gamera(0)
    s = g.download_state()
    assert (s["time"], s["otime"], s["dt"], s["ts"]) == (1.0, 1.0, dt, 5)
    assert np.array_equal(s["Gas"], gas) and np.array_equal(s["omagFlux"], mf)
