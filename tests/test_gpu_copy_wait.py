"""A wait of the flux and edge kernels for their copies to shared memory that runs
out: the step ends with a device error of its own, not with a time step failure, the
handle takes a new state, and the device goes on. The waits run out in the
bounds-check build, whose kernels are made to expect bytes that nothing sends
(GAM_COPY_STALL, read at gam_create)."""
import pytest

from mage_b200 import grids
from mage_b200.gamera import CHECK_LIB_PATH, GAM_ECUDA, GameraGPU, GamError, GamParams

pytestmark = pytest.mark.gpu

N = (16, 4, 4)


def _app(**kw):
    g = GameraGPU(GamParams(*N, **kw), lib_path=CHECK_LIB_PATH)
    g.set_geometry(grids.warped_periodic_corners(*N))
    g.init_blast_wave()
    return g


@pytest.mark.parametrize("fixed", [-1.0, 1e-4], ids=["cfl", "fixed"])
def test_a_wait_that_runs_out(monkeypatch, fixed):
    with monkeypatch.context() as m:
        m.setenv("GAM_COPY_STALL", "1")
        g = _app(fixedTimestep=fixed, strict=True)
    st = g.download_state()
    for _ in range(2):  # the step itself, and a call after it
        with pytest.raises(GamError, match="copy to shared memory") as ei:
            g.step_gamera(1)
        assert ei.value.code == GAM_ECUDA
    g.upload_state(st["Gas"], st["magFlux"], st["Bxyz"], st["oGas"], st["omagFlux"], st["time"], st["otime"], 1e-4)
    with pytest.raises(GamError, match="a step's copy to shared memory"):
        g.step_gamera(1)
    ok = _app(fixedTimestep=fixed, strict=True)
    ok.step_gamera(2)
    assert ok.bounds_status()["fired"] == 0
