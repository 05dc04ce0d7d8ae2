"""The whole step and its adjoint on grids whose extents are no multiples of the
flux and edge kernels' tiles (16 or 32 by 8 faces): the forward equals the PyTorch
restatement bit for bit, the adjoint autograd through it to 1e-12 (FP64) and 1e-5
(FP32), the bounds of the 16^3 case in test_gpu_wholestep.py."""
import numpy as np
import pytest
import torch

from mage_b200 import grids
from mage_b200.diffstep import DiffParams, Grid, WholeStep, step
from mage_b200.gamera import GameraGPU, GamParams

pytestmark = pytest.mark.gpu

DT = 5e-4
SIZES = [(24, 9, 13), (40, 17, 4), (16, 5, 10)]


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-12), (torch.float32, 1e-5)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("N", SIZES, ids=["x".join(map(str, n)) for n in SIZES])
def test_ragged_whole_step(N, dtype, tol):
    gpu = GameraGPU(GamParams(*N))
    gpu.set_geometry(grids.warped_periodic_corners(*N))
    gpu.init_blast_wave()
    st = gpu.download_state(old=False)
    g = Grid(DiffParams(*N), gpu.get_geometry_arrays(), dtype=dtype, device="cuda")
    rng = np.random.default_rng(23)

    def noise(shape):
        return torch.as_tensor(rng.standard_normal(shape), device="cuda").to(dtype)
    Gas0 = g.cell_box(st["Gas"]) * (1 + 1e-3 * noise((5,) + tuple(g.face.shape[1:])))
    mf0 = g.face_box(st["magFlux"]) + 1e-3 * g.face * noise(g.face.shape)
    with torch.no_grad():
        old = {"Gas": Gas0, "mf": mf0, "B": g.bxyz(mf0)}
        cur = step(g, old, old, DT, DT)
    leaves = [t.detach().clone().requires_grad_(True) for t in (cur["Gas"], cur["mf"], old["Gas"], old["mf"])]
    with torch.enable_grad():
        c = {"Gas": leaves[0], "mf": leaves[1], "B": g.bxyz(leaves[1])}
        o = {"Gas": leaves[2], "mf": leaves[3], "B": g.bxyz(leaves[3])}
        ref = step(g, c, o, DT, DT)
        dn = {k: noise(ref[k].shape) for k in ("Gas", "mf", "B")}
        dref = torch.autograd.grad([ref[k] for k in dn], leaves, list(dn.values()))
    ws = WholeStep(g)
    out = ws.forward(cur, old, DT, DT)
    for k in ("Gas", "mf", "B"):
        assert torch.equal(out[k], ref[k].detach()), (k, float((out[k] - ref[k]).abs().max()))
    kept = ws.adjoint(cur, old, DT, DT, dn, saved=True)
    again = ws.adjoint(cur, old, DT, DT, dn)
    num = sum(float((x - y).norm()) ** 2 for x, y in zip(kept, dref)) ** 0.5
    den = sum(float(y.norm()) ** 2 for y in dref) ** 0.5
    assert num <= tol * den, num / den
    for a, b in zip(kept, again):
        assert torch.equal(a, b), float((a - b).abs().max())


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["fp64", "fp32"])
def test_one_array_for_both_adjoints(dtype):
    """A start whose State is its oState: with one array given for both adjoints, the
    adjoint adds both into it."""
    N = (24, 9, 13)
    gpu = GameraGPU(GamParams(*N))
    gpu.set_geometry(grids.warped_periodic_corners(*N))
    gpu.init_blast_wave()
    st = gpu.download_state(old=False)
    g = Grid(DiffParams(*N), gpu.get_geometry_arrays(), dtype=dtype, device="cuda")
    gas, mf = g.cell_box(st["Gas"]), g.face_box(st["magFlux"])
    cur = {"Gas": gas, "mf": mf, "B": g.bxyz(mf)}
    gen = torch.Generator(device="cuda").manual_seed(3)
    dn = {k: torch.randn(cur[k].shape, generator=gen, dtype=dtype, device="cuda") for k in ("Gas", "mf")}
    ws = WholeStep(g)
    ws.forward(cur, cur, DT, DT)
    d = ws.adjoint(cur, cur, DT, DT, dn, saved=True)
    zG, zM = torch.zeros_like(gas), torch.zeros_like(mf)
    both = ws.adjoint(cur, cur, DT, DT, dn, [zG, zM, zG, zM], saved=True)
    assert torch.equal(both[0], d[0] + d[2]) and torch.equal(both[1], d[1] + d[3])
