"""A handle that does not fit the device beside the memory that PyTorch's allocator
keeps for later tensors is created after that has been given back (a stand-in for the
library; no GPU)."""
import pytest
import torch

from mage_b200 import gamera
from mage_b200.gamera import GAM_ECUDA, GAM_EINVAL, GameraGPU, GamError, GamParams


class Library:
    """gam_create fails with the given codes and messages in turn, then succeeds."""

    def __init__(self, *fails):
        self.fails, self.live, self.made = list(fails), set(), 0

    def gam_create(self, p, out):
        self.made += 1
        out._obj.value = self.made
        self.live.add(self.made)
        self.rc, self.msg = self.fails.pop(0) if self.fails else (0, b"")
        return self.rc

    def gam_last_error(self, h):
        assert h.value in self.live
        return self.msg

    def gam_destroy(self, h):
        self.live.remove(h.value)


NO_MEMORY = (GAM_ECUDA, b"cudaMalloc failed (out of device memory?)")


@pytest.mark.parametrize("cached", [True, False])
@pytest.mark.parametrize("fails", [(), (NO_MEMORY,), (NO_MEMORY, NO_MEMORY), ((GAM_EINVAL, b"nG must be 4"),)])
def test_create_again_without_the_cache(monkeypatch, fails, cached):
    lib, given = Library(*fails), []
    monkeypatch.setattr(gamera, "load_library", lambda path: lib)
    monkeypatch.setattr(torch.cuda, "is_initialized", lambda: cached)
    monkeypatch.setattr(torch.cuda, "empty_cache", lambda: given.append(1))
    again = bool(fails) and fails[0] is NO_MEMORY and cached
    if len(fails) > (1 if again else 0):
        with pytest.raises(GamError) as ei:
            GameraGPU(GamParams(16, 4, 4))
        assert ei.value.code == fails[0][0]
        del ei
    else:
        g = GameraGPU(GamParams(16, 4, 4))
        assert g.h.value == lib.made and lib.live == {lib.made}
        g.close()
    assert len(given) == again and lib.made == 1 + again
