"""The strict form's second try: cells with momenta and face fluxes of 1e-145 to
1e-200, outside the range of the quotients without a branch (2^-450), among ordinary
ones. Their work is done again with divisions, and the whole box equals the CPU
restatement bit for bit, with AB2 and AB3, in 2.5-D and around a pole with a ring."""
import numpy as np
import pytest

from mage_b200 import grids
from mage_b200.gamera import BC_LFM, BC_PERIODIC, BC_SPHIN, BC_ZEROGRAD, GameraGPU, GamParams
from oracle.oracle import Oracle, OracleParams
from tests.helpers import gpu_from_oracle, make_oracle, rel_err

pytestmark = pytest.mark.gpu

RINGS = (BC_SPHIN, BC_ZEROGRAD, BC_LFM, BC_LFM, BC_PERIODIC, BC_PERIODIC)


def _make_small(o, rng):
    """Tiny values of either sign in a third of the cells and faces of State and oState."""
    def tiny(shape):
        return rng.choice([-1.0, 1.0], shape) * 10.0 ** rng.uniform(-200, -145, shape)
    for name in ("Gas", "oGas"):
        for v in (1, 2, 3):
            a = o.array(name)[v]
            a[...] = np.where(rng.uniform(size=a.shape) < 1 / 3, tiny(a.shape), a)
    for name in ("magFlux", "omagFlux"):
        a = o.array(name)[2]
        a[...] = np.where(rng.uniform(size=a.shape) < 1 / 3, tiny(a.shape), a)


@pytest.mark.parametrize("case", ["ab2", "ab3", "2.5-D", "ring"])
def test_out_of_range_operands(oracle_built, case):
    rng = np.random.default_rng(17)
    if case == "ring":
        N = (16, 16, 16)
        xyz = grids.lfm_corners(*N, th0=0.01)
        o = Oracle(OracleParams(*N, bc=RINGS, ringNch=(8,)), xyz, "gm")
        o.ic_blast_wave(x0=6.0, y0=0.7, z0=0.0, rC=3.0, B0=0.3)
        assert o.init_finish() == 0
        _make_small(o, rng)
        g = GameraGPU(GamParams(*N, bc=RINGS, strict=True))
        g.set_rings((8,))
        g.set_geometry(xyz)
        sc = o.scalars()
        g.upload_state(o.array("Gas"), o.array("magFlux"), o.array("Bxyz"), o.array("oGas"), o.array("omagFlux"),
                       sc["time"], sc["otime"], sc["dt"], sc["ts"])
    else:
        kw = {"doAB3": case == "ab3"}
        o, _ = make_oracle("ot" if case == "2.5-D" else "bw", (24, 9, 1 if case == "2.5-D" else 12), variant="gm", **kw)
        _make_small(o, rng)
        g = gpu_from_oracle(o, strict=True, **kw)
        if case == "ab3":
            g.set_oostate(o.array("oomagFlux"), o.scalars()["ootime"])
    for n in (1, 2):
        assert o.step(n) == 0
        g.step_gamera(n)
        s = g.download_state()
        for k in ("Gas", "magFlux", "Bxyz"):
            assert np.array_equal(s[k], o.array(k)), (n, k, rel_err(s[k], o.array(k)), int((s[k] != o.array(k)).sum()))
