"""The sweep with as many kept work areas as its memory bound gives: one (every
other step of a segment runs forward once more inside its adjoint), fewer than a
segment has steps, one for each; a last segment shorter than the others. The loss
and the gradients have the same bits: the adjoint of kept intermediates and of
recomputed ones takes the same values."""
import pytest
import torch

from mage_b200.diffstep import WholeStep, loss_and_grad_c
from tests.test_gpu_wholestep import DT, PERIODIC, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("nsteps,seg", [(7, 3), (4, 4), (3, 1)])
def test_sweep_does_not_depend_on_the_areas(monkeypatch, nsteps, seg, dtype):
    g, Gas0, mf0, _ = _setup(PERIODIC, dtype, 11)
    every = WholeStep.work_areas
    res = []
    for n in (1, 2, 8):
        monkeypatch.setattr(WholeStep, "work_areas", lambda self, k, n=n: every(self, min(k, n)))
        res.append(loss_and_grad_c(g, Gas0, mf0, DT, nsteps, seg=seg))
    for L, gG, gF in res[1:]:
        assert L == res[0][0]
        assert torch.equal(gG, res[0][1]) and torch.equal(gF, res[0][2])
