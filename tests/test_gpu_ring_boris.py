"""Rings about the LFM axis with the Boris correction, whose step takes the ring
average after the cell update (CellBoris looks at the field before it): the strict
build equals the CPU restatement bit for bit, an off-axis blast wave and the
magnetosphere with its hooks."""
import numpy as np
import pytest

from mage_b200 import dipole, grids
from mage_b200.gamera import BACKGROUND_ARRAYS, GameraGPU, GamParams
from oracle.oracle import Oracle, OracleParams
from tests.test_gpu_ring import BCS, BW, DTCPL, MBCS, WIND, _bitwise, _fields

pytestmark = pytest.mark.gpu

BORIS = {"doBoris": True, "Ca": 10.0}


def test_blast_with_rings_and_boris(oracle_built):
    N = (16, 16, 16)
    xyz = grids.lfm_corners(*N, th0=0.01)
    o = Oracle(OracleParams(*N, bc=BCS, ringNch=(8,), **BORIS), xyz, "gm")
    o.ic_blast_wave(**BW)
    assert o.init_finish() == 0
    g = GameraGPU(GamParams(*N, bc=BCS, strict=True, **BORIS))
    g.set_rings((8,))
    g.set_geometry(xyz)
    g.init_blast_wave(**BW)
    for nst in (1, 5):
        assert o.step(nst) == 0
        g.step_gamera(nst)
        _bitwise(o, g, nst)


def test_magnetosphere_with_rings_and_boris(oracle_built):
    N = (16, 8, 16)
    xyz = grids.lfm_corners(*N, th0=0.01)
    E, Ee = _fields(N)
    o = Oracle(OracleParams(*N, doBackground=True, M0=dipole.M0, wind=WIND, bc=MBCS, ringNch=(8,), **BORIS), xyz, "gm")
    o.set_ionosphere(E, Ee, dipole.M0, DTCPL, True, 2)
    o.ic_dipole_wind(0.01, 31337)
    assert o.init_finish() == 0
    g = GameraGPU(GamParams(*N, doBackground=1, bc=MBCS, strict=True, **BORIS))
    g.set_rings([8])
    g.set_geometry(xyz)
    g.set_background({n: o.array(n) for n, _ in BACKGROUND_ARRAYS})
    g.set_ionosphere(E, Ee, dipole.M0, DTCPL, True, 2)
    g.init_dipole_wind(WIND, 31337, 0.01)
    for nst in (1, 5):
        assert o.step(nst) == 0
        g.step_gamera(nst)
        _bitwise(o, g, nst)
