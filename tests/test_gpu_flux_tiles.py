"""The flux kernels' shared-memory tiles (16 or 32 faces by 8) at sizes
around them: one tile and less, whole tiles, remainders in every direction, a
2.5-D grid; both reconstructions, the limiter on either state, no field. The
strict build equals the CPU restatement bit for bit; FP32 stays within its
rounding: 2e-6 relative to the largest value after 3 steps (the differences of
this step measure 1e-7 to 5e-7)."""
import numpy as np
import pytest

from mage_b200.gamera import FP32
from tests.helpers import gpu_from_oracle, make_oracle, rel_err

pytestmark = pytest.mark.gpu

SIZES = [(16, 4, 4), (16, 7, 9), (24, 8, 8), (32, 9, 15), (40, 17, 12), (32, 31, 1)]


@pytest.mark.parametrize("kw", [{}, {"up7": True}, {"doLFMLim": False}, {"doMHD": False}],
                         ids=["8cent", "7up", "nolfmlim", "hydro"])
@pytest.mark.parametrize("N", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
def test_tiles_match_oracle(oracle_built, N, kw):
    o, _ = make_oracle("ot" if N[2] == 1 else "bw", N, variant="gm", **kw)
    g = gpu_from_oracle(o, strict=True)
    f = gpu_from_oracle(o, precision=FP32)
    assert o.step(3) == 0
    g.step_gamera(3)
    f.step_gamera(3)
    s, s32 = g.download_state(), f.download_state()
    # without a field the step leaves magFlux and Bxyz alone, which the two sides start differently
    for k in ("Gas", "magFlux", "Bxyz") if kw.get("doMHD", True) else ("Gas",):
        assert np.array_equal(s[k], o.array(k)), (N, kw, k, rel_err(s[k], o.array(k)))
        assert rel_err(s32[k], o.array(k)) <= 2e-6, (N, kw, k, rel_err(s32[k], o.array(k)))
