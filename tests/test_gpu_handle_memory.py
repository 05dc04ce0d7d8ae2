"""A handle's device memory: the values per position of the padded box that a grid
takes in each form. The bounds are what the forms took before the reconstructions'
tables (gam_geom_tables) came to them, so that a grid that fitted a device then
still does: 179 FP64 values (24 more with a background field; FP32 has 92 beside 191
of its own) and a transfer buffer of 27 FP64 face values."""
import pytest
import torch

from mage_b200.gamera import FP32, GameraGPU, GamParams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,doubles,floats", [
    (dict(strict=True), 179, 0), (dict(strict=True, doLFMLim=False), 179, 0), (dict(), 179, 0),
    (dict(strict=True, doBackground=True), 203, 0), (dict(precision=FP32), 92, 191),
], ids=["strict", "strict-nolfmlim", "fma", "background", "fp32"])
def test_a_handle_takes_no_more(kw, doubles, floats):
    N = (128, 96, 96)
    sx, pos = N[0] + 16, (N[1] + 9) * (N[2] + 9)
    GameraGPU(GamParams(16, 4, 4)).close()  # the context and the library's kernels
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    g = GameraGPU(GamParams(*N, **kw))
    took = free - torch.cuda.mem_get_info()[0]
    g.close()
    limit = sx * pos * (8 * doubles + 4 * floats) + (N[0] + 9) * pos * 8 * 27
    # each of the 50 arrays is an allocation of its own, in units of 2 MiB (a table more
    # of 12 values is 145 MiB)
    assert took <= limit + 75 * (1 << 20), (took / 2**20, limit / 2**20)
