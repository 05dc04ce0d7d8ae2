"""The memory of the checkpointed sweep's kept work areas (loss_and_grad_c), on the
CPU with a linear stand-in for the step: it takes fewer areas when the memory for
them is not there, and runs without any when they leave too little for the rest, with
the same loss and gradients, which are those of autograd. A kept area is asked for
the step whose intermediates it holds."""
import types

import pytest
import torch

from mage_b200 import diffstep
from mage_b200.diffstep import WholeStep, loss_and_grad_c

A, B = 1.25, -0.375  # the next State is A State + B oState


class Linear(WholeStep):
    """WholeStep with a linear step; memory: how many areas fit, and how many leave
    room for the sweep."""
    fit, room = 99, 99

    def __init__(self, g):
        self.g, self.holds, self.calls = g, {}, 0
        self.work = torch.zeros(8, dtype=torch.uint8)

    def forward(self, cur, old, dt, odt, work=None):
        self.calls += 1
        if work is not None and self.kept > self.room and self.calls >= 2:  # kept areas are held
            raise torch.OutOfMemoryError("no room")
        self.holds[id(self.work if work is None else work)] = (cur["Gas"].clone(), old["Gas"].clone())
        nxt = {k: A * cur[k] + B * old[k] for k in ("Gas", "mf")}
        return nxt | {"B": 2 * nxt["mf"]}

    def adjoint(self, cur, old, dt, odt, dnxt, acc=None, saved=False, dinflow=None, work=None):
        if saved:
            c, o = self.holds[id(self.work if work is None else work)]
            assert torch.equal(c, cur["Gas"]) and torch.equal(o, old["Gas"])
        d = dict(dnxt)
        if "B" in d:
            d["mf"] = d["mf"] + 2 * d["B"]
        out = [acc[0] + A * d["Gas"], acc[1] + A * d["mf"], acc[2] + B * d["Gas"], acc[3] + B * d["mf"]]
        return out

    def work_areas(self, n):
        real = torch.empty_like
        left = [self.fit - 1]

        def few(t, *a, **k):
            if t is self.work:
                if left[0] == 0:
                    raise torch.OutOfMemoryError("no piece")
                left[0] -= 1
            return real(t, *a, **k)
        torch.empty_like = few
        try:
            areas = WholeStep.work_areas(self, n)
        finally:
            torch.empty_like = real
        self.kept = len(areas)
        return areas


def _loss(g, s):
    return (s["Gas"] ** 2).sum() + (s["B"] ** 3).sum() + s["mf"].sum()


@pytest.mark.parametrize("nsteps,seg", [(7, 3), (4, 4), (3, 1), (5, None)])
@pytest.mark.parametrize("fit,room", [(99, 99), (2, 99), (1, 99), (99, 1), (1, 0), (99, 0)])
def test_sweep_within_its_memory(monkeypatch, nsteps, seg, fit, room):
    monkeypatch.setattr(diffstep, "WholeStep", Linear)
    monkeypatch.setattr(Linear, "fit", fit)
    monkeypatch.setattr(Linear, "room", room)
    g = types.SimpleNamespace(dtype=torch.float64, inflow=None, bxyz=lambda mf: 2 * mf)
    gen = torch.Generator().manual_seed(3)
    gas = torch.randn((5, 2, 3, 4), generator=gen, dtype=torch.float64)
    mf = torch.randn((3, 2, 3, 4), generator=gen, dtype=torch.float64)
    L, dG, dF = loss_and_grad_c(g, gas, mf, 1.0, nsteps, seg=seg, lossf=_loss)
    G, M = gas.clone().requires_grad_(True), mf.clone().requires_grad_(True)
    cur = old = {"Gas": G, "mf": M}
    for _ in range(nsteps):
        cur, old = {k: A * cur[k] + B * old[k] for k in cur}, cur
    ref = _loss(g, cur | {"B": 2 * cur["mf"]})
    rG, rF = torch.autograd.grad(ref, [G, M])
    ref = float(ref.detach())
    assert abs(L - ref) <= 1e-12 * abs(ref)
    assert torch.allclose(dG, rG, rtol=1e-12) and torch.allclose(dF, rF, rtol=1e-12)


def test_areas_leave_the_sweeps_own_memory(monkeypatch):
    ws = WholeStep.__new__(WholeStep)
    ws.work = types.SimpleNamespace(is_cuda=True, device="cuda:0", numel=lambda: 1 << 30)
    free, held, asked = [100 << 30], [4 << 30], []
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d: asked.append(1) or (free[0], 180 << 30))
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda d: {
        "reserved_bytes": {"all": {"current": held[0] + (3 << 30)}}, "allocated_bytes": {"all": {"current": 3 << 30}}})
    assert ws.areas_that_fit(99) == 17                 # 16 GiB
    assert ws.areas_that_fit(99, 64 << 30) == 11       # a quarter of 40 GiB
    assert ws.areas_that_fit(99, 200 << 30) == 1
    assert ws.areas_that_fit(6) == 6 and len(asked) == 4
    assert ws.areas_that_fit(5) == 5 and len(asked) == 4   # what the allocator holds
    free[0] = 0
    assert ws.areas_that_fit(6) == 2                   # a quarter of 4 GiB, of the allocator's own
    assert ws.areas_that_fit(5, 1) == 1
    held[0] = 30 << 30
    assert ws.areas_that_fit(99, 14 << 30) == 17 and len(asked) == 6
    held[0] = 0
    ws.work.numel = lambda: 1 << 28
    assert ws.areas_that_fit(5, 99 << 30) == 5 and len(asked) == 6  # 1 GiB: not looked at
    assert ws.areas_that_fit(6, 99 << 30) == 1
