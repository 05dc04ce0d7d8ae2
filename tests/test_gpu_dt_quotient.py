"""CalcDT's sound speed in the forms that multiply by reciprocals is that of a
division: for a uniform gas at rest, without a field, dt = CFL dl / sqrt(gamma P / rho)
has one rounding per operation, so the value is known to the last bit."""
import numpy as np
import pytest

from mage_b200 import grids
from mage_b200.gamera import FP32, GameraGPU, GamParams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, FP32], ids=["fma", "fp32"])
def test_sound_speed_is_a_quotient(precision):
    N = (16, 4, 4)
    f = np.float32 if precision == FP32 else np.float64
    g = GameraGPU(GamParams(*N, precision=precision, doMHD=False))
    g.set_geometry(grids.uniform_corners(*N))
    geo = g.get_geometry_arrays()
    # the cells of CalcDT's range; FP32 keeps dl in single precision
    dl = np.minimum(np.minimum(geo["di"], geo["dj"]), geo["dk"])[0, 3:-3, 3:-3, 3:-3].astype(f).astype(np.float64).min()
    gam, cfl = 5.0 / 3.0, 0.3
    mf = np.zeros(g.shape("face", 3))
    rng = np.random.default_rng(5)
    off = []
    for _ in range(64):
        rho, E = (float(f(q)) for q in 10.0 ** rng.uniform(-3, 3, 2))
        gas = np.zeros(g.shape("cell", 5))
        gas[0], gas[4] = rho, E
        g.upload_state(gas, mf, None, gas, mf, 0.0, -1.0, 1.0)
        cs = np.sqrt(gam * ((gam - 1.0) * E) / rho)
        dt = cfl * dl / np.sqrt(cs * cs)
        got = g.calc_dt()
        if got != dt:
            off.append((rho, E, (got - dt) / dt))
    assert not off, (len(off), off[:4])
