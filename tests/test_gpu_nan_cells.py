"""A cell that is not a number, under a fixed time step (no CalcDT stops the run): how
far it spreads is given by the limiter's comparisons (recon.F90:231-301). The strict
build's whole box equals the CPU restatement's, NaN for NaN, and the FP32 form has
NaN in the same places."""
import numpy as np
import pytest

from mage_b200.gamera import FP32
from tests.helpers import gpu_from_oracle, make_oracle

pytestmark = pytest.mark.gpu

DT = 1.0e-4


@pytest.mark.parametrize("kw", [{}, {"up7": True}, {"doLFMLim": False}, {"up7": True, "doLFMLim": False}],
                         ids=["8cent", "7up", "8cent-nolfmlim", "7up-nolfmlim"])
def test_nan_spreads_as_in_the_restatement(oracle_built, kw):
    o, _ = make_oracle("bw", (24, 12, 13), variant="gm", fixedTimestep=True, fixedDT=DT, **kw)
    assert o.step(1) == 0
    for name in ("Gas", "oGas"):
        o.array(name)[:, 10, 9, 14] = np.nan
        o.array(name)[3, 7, 7, 9] = -np.nan
    o.array("magFlux")[1, 12, 12, 20] = o.array("omagFlux")[1, 12, 12, 20] = np.nan
    g = gpu_from_oracle(o, strict=True, fixedTimestep=DT)
    f = gpu_from_oracle(o, precision=FP32, fixedTimestep=DT)
    for n in (1, 1):
        o.step(n)
        g.step_gamera(n)
        f.step_gamera(n)
        s, s32 = g.download_state(), f.download_state()
        for k in ("Gas", "magFlux", "Bxyz"):
            assert np.array_equal(s[k], o.array(k), equal_nan=True), (k, int((np.isnan(s[k]) != np.isnan(o.array(k))).sum()))
            d = np.isnan(s32[k]) != np.isnan(o.array(k))
            assert not d.any(), (k, "fp32", int(d.sum()), int(np.isnan(o.array(k)).sum()))
