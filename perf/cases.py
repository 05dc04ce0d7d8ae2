"""The work that a user of the step has it do, as cases to be timed and compared.

A case is one of four uses of the public entry points:

* ``forward``: a simulation that runs on the device and writes its output
  every few steps (``GameraGPU.step_gamera`` + ``download_state``), in the
  FP64 drop-in ("strict"), the FP64 FMA form and the FP32 form;
* ``dropin``: the Fortran driver's loop around ``AdvanceModel``: State goes up,
  one step, State comes back (``upload_state``, ``advance_model``,
  ``download_state``);
* ``sweep``: the gradient of a loss after some steps with respect to the start
  (``diffstep.loss_and_grad_c``);
* ``adjoint``: one whole step and its adjoint (``diffstep.WholeStep``).

The problems and their sizes are those of the decks, the benchmark and the
tests: the Orszag-Tang vortex, the blast wave on the warped periodic grid, the
dipole in a solar wind on a spherical grid, and the magnetosphere on an
LFM-style grid with its ionospheric boundary and ring average. The seed moves
the vortex and the blast, and draws the wind's density noise.
"""
import math

import numpy as np
import torch

from mage_b200 import dipole, grids, workloads
from mage_b200.diffstep import DiffParams, Grid, WholeStep, loss_and_grad_c
from mage_b200.gamera import FP32, FP64, RECON_7UP, RECON_8CENT, GameraGPU, GamParams

NG = 4
PI = math.pi


def _case(name, kind, problem, n, form, steps, recon="8cent", option="none"):
    return {"name": name, "kind": kind, "problem": problem, "ni": n[0], "nj": n[1], "nk": n[2], "form": form,
            "steps": steps, "recon": recon, "option": option}


def listed():
    return [
        # the smallest deck (2.5-D vortex on 32 x 32), a line of output every 10 steps
        _case("ot32_2d_strict", "forward", "ot", (32, 32, 1), "strict", 10),
        # the vortex the reference's parity is quoted on, its 100 steps
        _case("ot128_strict", "forward", "ot", (128, 128, 4), "strict", 100),
        # a ragged grid with the other reconstruction
        _case("blast_ragged_7up_fma", "forward", "blast", (72, 53, 41), "fma", 10, recon="7up"),
        # an ordinary single-precision run
        _case("blast64_fp32", "forward", "blast", (64, 64, 64), "fp32", 20),
        # the headline grid in the three forms
        _case("blast192_strict", "forward", "blast", (192, 192, 192), "strict", 10),
        _case("blast192_fma", "forward", "blast", (192, 192, 192), "fma", 10),
        _case("blast192_fp32", "forward", "blast", (192, 192, 192), "fp32", 10),
        # background field, inner sphere, solar wind: the precision form's workload
        _case("dipole96_fp32", "forward", "dipole", (96, 96, 128), "fp32", 20),
        # the magnetosphere: ionospheric boundary with its hooks, rings about the axis
        _case("lfm96_strict", "forward", "lfm", (96, 96, 128), "strict", 10),
        # the Fortran driver's loop: the state crosses the host boundary every step
        _case("dropin96_strict", "dropin", "blast", (96, 96, 96), "strict", 1),
        # the gradient of the blast-wave loss over 20 steps
        _case("sweep64_fp64", "sweep", "blast", (64, 64, 64), "fp64", 20),
        # one step of a sweep, forward and back, on a larger grid. The gradients are
        # in FP64: a limiter's switch that a rounding decides turns single values of
        # an FP32 gradient over, so those cannot be compared one by one
        _case("adjoint128_fp64", "adjoint", "blast", (128, 128, 128), "fp64", 1),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of its range, odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sizes(rng, lo, hi):
    """Three sizes; the I size is a multiple of 8, as the grid asks."""
    return [8 * max(2, round(_size(rng, lo, hi) / 8)), _size(rng, lo, hi), _size(rng, lo, hi)]


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "forward", "dropin", "sweep", "adjoint"])
    if kind in ("sweep", "adjoint"):
        n = _sizes(rng, 16, 96)
        steps = rng.choice([4, 6, 9]) if kind == "sweep" else 1
        return _case("drawn", kind, "blast", n, "fp64", steps)
    if kind == "dropin":
        n = _sizes(rng, 16, 110)
        return _case("drawn", kind, "blast", n, rng.choice(["strict", "fma", "fp32"]), 1)
    problem = rng.choice(["ot", "blast", "blast", "dipole", "lfm"])
    form = rng.choice(["strict", "fma", "fp32"])
    recon, option = "8cent", "none"
    if problem == "ot":
        n = _sizes(rng, 16, 256)[:2] + [rng.choice([1, 1, 4, 8])]
        steps = rng.choice([10, 20, 50])
        form = rng.choice(["strict", "fma"])
        option = rng.choice(["none", "none", "ab3"])
    elif problem == "blast":
        n = _sizes(rng, 16, 160)
        steps = rng.choice([2, 5, 10])
        recon = rng.choice(["8cent", "8cent", "7up"])
        option = rng.choice(["none", "none", "nolfmlim", "boris", "ab3"])
    elif problem == "dipole":
        n = _sizes(rng, 24, 112)
        steps = rng.choice([5, 10])
        option = rng.choice(["none", "boris"])
    else:  # the default rings exist for these numbers of cells around the axis
        n = _sizes(rng, 32, 112)[:2] + [rng.choice([64, 128])]
        steps = rng.choice([5, 10])
    return _case("drawn", kind, problem, n, form, steps, recon, option)


# ----------------------------------------------------------------- inputs
def _n(case):
    return int(case["ni"]), int(case["nj"]), int(case["nk"])


_corner_cache = {}  # the grid file a program has read: the same for every seed


def _corners(case):
    key = (case["problem"],) + _n(case)
    if key not in _corner_cache:
        if len(_corner_cache) > 6:
            _corner_cache.clear()
        if case["problem"] == "ot":
            xyz = grids.uniform_corners(*_n(case))
        elif case["problem"] == "blast":
            xyz = grids.warped_periodic_corners(*_n(case))
        elif case["problem"] == "dipole":
            xyz = grids.spherical_corners(*_n(case))
        else:
            xyz = grids.lfm_corners(*_n(case), th0=0.01)
        _corner_cache[key] = xyz
    return _corner_cache[key]


def _blast(seed):
    """Centre, pressure ratio and radius of the blast."""
    r = np.random.default_rng(1000 + seed)
    c = 0.5 + 0.1 * r.uniform(-1, 1, 3)
    return {"x0": float(c[0]), "y0": float(c[1]), "z0": float(c[2]), "pRat": float(r.uniform(80, 120)),
            "rC": float(r.uniform(0.1, 0.14))}


def _vortex(case, seed):
    """The Orszag-Tang start with seeded phases, as the driver's arrays with
    their ghosts; uniform unit box, face fluxes field times area."""
    n = _n(case)
    ph = 2 * PI * np.random.default_rng(2000 + seed).uniform(0, 1, 4)
    d = [1.0 / q for q in n]

    def at(q, half, m):
        return (np.arange(-NG, n[q] + NG + m) + half) * d[q]
    xc, yc = at(0, 0.5, 0), at(1, 0.5, 0)
    nk = n[2] + 2 * NG
    rho, p0, b0 = 25 / (36 * PI), 5 / (12 * PI), 1 / math.sqrt(4 * PI)
    vx = -np.sin(2 * PI * yc + ph[0])[None, :, None] + np.zeros((nk, 1, xc.size))
    vy = np.sin(2 * PI * xc + ph[1])[None, None, :] + np.zeros((nk, yc.size, 1))
    gas = np.zeros((5, nk, yc.size, xc.size))
    gas[0] = rho
    gas[1], gas[2] = rho * vx, rho * vy
    gas[4] = 0.5 * rho * (vx * vx + vy * vy) + p0 / (5.0 / 3.0 - 1)
    mf = np.zeros((3, nk + 1, yc.size + 1, xc.size + 1))
    mf[0, :-1, :-1] = (-b0 * np.sin(2 * PI * yc + ph[2]) * d[1] * d[2])[None, :, None]
    mf[1, :-1, :, :-1] = (b0 * np.sin(4 * PI * xc + ph[3]) * d[0] * d[2])[None, None, :]
    return gas, mf


def _params(case):
    kw = {"precision": FP32 if case["form"] == "fp32" else FP64, "strict": case["form"] == "strict",
          "rmeth": RECON_7UP if case["recon"] == "7up" else RECON_8CENT}
    if case["option"] == "boris":
        kw.update(doBoris=True, Ca=10.0)
    if case["option"] == "ab3":
        kw.update(doAB3=True)
    if case["option"] == "nolfmlim":
        kw.update(doLFMLim=False)
    if case["problem"] == "ot":
        kw.update(do25D=case["nk"] == 1)
    if case["problem"] == "dipole":
        kw.update(doBackground=True, bc=workloads.DIPOLE_BCS)
    if case["problem"] == "lfm":
        kw.update(doBackground=True, bc=workloads.MAGSPHERE_BCS)
    return GamParams(*_n(case), **kw)


def _app(case, seed):
    """The program's handle with its grid and start."""
    g = GameraGPU(_params(case))
    if case["problem"] == "lfm":
        g.set_rings()
    g.set_geometry(_corners(case))
    if case["problem"] == "ot":
        gas, mf = _vortex(case, seed)
        g.upload_state(gas, mf, None, gas, mf, 0.0, -1.0, 1.0)
        dt = g.calc_dt()
        g.upload_state(gas, mf, None, gas, mf, 0.0, -dt, dt)
    elif case["problem"] == "blast":
        g.init_blast_wave(**_blast(seed))
    else:
        g.set_background_dipole(dipole.M0)
        if case["problem"] == "lfm":
            e, ee = workloads.ion_fields(_n(case))
            g.set_ionosphere(e, ee, dipole.M0, workloads.ION_DTCPL, True, 1)
            g.init_dipole_wind(dipole.wind_code_units(), seed=seed)
        else:
            wind = dipole.wind_code_units()
            g.set_wind(wind)
            g.init_dipole_wind(wind, seed=seed)
    return g


def _pinned(g, names):
    kinds = {"Gas": ("cell", 5), "magFlux": ("face", 3), "Bxyz": ("cell", 3)}
    return {k: torch.empty(g.shape(*kinds[k]), dtype=torch.float64, pin_memory=True).numpy() for k in names}


_geo_cache = {}  # metric arrays of the differentiation form's grid, as read from the driver


def _diff_grid(case):
    """(Grid, start Gas and magFlux of the unmoved blast, its dt)."""
    n = _n(case)
    if n not in _geo_cache:
        if len(_geo_cache) > 2:
            _geo_cache.clear()
        g = GameraGPU(GamParams(*n))
        g.set_geometry(_corners(case))
        _geo_cache[n] = g.get_geometry_arrays()
        g.close()
    g = GameraGPU(GamParams(*n))
    g.set_geometry(_corners(case))
    dtype = torch.float32 if case["form"] == "fp32" else torch.float64
    return g, Grid(DiffParams(*n), _geo_cache[n], dtype=dtype, device="cuda")


def _noise(shape, seed, dtype):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3000 + seed)
    return torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda").to(dtype)


def _noises(n, seed, dtype):
    """Noise on a State's Gas and magFlux: the cells and faces that the box holds."""
    size = tuple(q + 2 * NG + 1 for q in n[::-1])
    gas, mf = _noise((5,) + size, seed, dtype), _noise((3,) + size, seed + 7, dtype)
    for q in range(3):
        last = (slice(None),) * q + (-1,)
        gas[(slice(None), *last)] = 0
        for d in range(3):
            if d != 2 - q:
                mf[(d, *last)] = 0
    return gas, mf


def _still(dtype, device="cuda"):
    """The scale of the noise on the momentum of a gas at rest."""
    return torch.tensor([0.0, 1.0, 1.0, 1.0, 0.0], dtype=dtype, device=device).reshape(5, 1, 1, 1)


def prepare(case, seed):
    if case["kind"] in ("forward", "dropin"):
        g = _app(case, seed)
        if case["kind"] == "forward":
            return {"case": case, "app": g, "out": _pinned(g, ("Gas", "magFlux", "Bxyz"))}
        names = ("Gas", "magFlux")
        st = g.download_state(_pinned(g, names), names=names)
        return {"case": case, "app": g, "in": st, "out": _pinned(g, names), "dt": st["dt"]}
    app, grid = _diff_grid(case)
    app.init_blast_wave(**_blast(seed))
    st = app.download_state(old=False)
    app.close()
    # 1e-3 noise on the start, as the gradient benchmark has it
    gas, mf = grid.cell_box(st["Gas"]), grid.face_box(st["magFlux"])
    ngas, nmf = _noises(_n(case), seed, grid.dtype)
    gas, mf = gas + 1e-3 * (gas + _still(grid.dtype)) * ngas, mf + 1e-3 * grid.face * nmf
    s = {"case": case, "grid": grid, "gas": gas, "mf": mf, "dt": 0.5 * st["dt"]}
    if case["kind"] == "adjoint":
        s["ws"] = WholeStep(grid)
        old = {"Gas": gas, "mf": mf, "B": grid.bxyz(mf)}
        s["old"], s["cur"] = old, s["ws"].forward(old, old, s["dt"], s["dt"])
        # the adjoint a later step hands back
        s["dn"] = dict(zip(("Gas", "mf"), _noises(_n(case), seed + 11, grid.dtype)))
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "forward":
        dt, t = s["app"].step_gamera(case["steps"])
        return dict(s["app"].download_state(s["out"], names=("Gas", "magFlux", "Bxyz")))
    if case["kind"] == "dropin":
        g, st = s["app"], s["in"]
        # the whole State and oState of the driver: the same start every pass
        g.upload_state(st["Gas"], st["magFlux"], None, st["Gas"], st["magFlux"], 0.0, -s["dt"], s["dt"])
        for _ in range(case["steps"]):
            g.advance_model(0.0)
        return dict(g.download_state(s["out"], names=("Gas", "magFlux")))
    if case["kind"] == "sweep":
        loss, dgas, dmf = loss_and_grad_c(s["grid"], s["gas"], s["mf"], s["dt"], case["steps"])
        return {"loss": loss, "dGas": dgas, "dmagFlux": dmf}
    ws, dt = s["ws"], s["dt"]
    nxt = ws.forward(s["cur"], s["old"], dt, dt)
    d = ws.adjoint(s["cur"], s["old"], dt, dt, s["dn"], saved=True)
    return {"Gas": nxt["Gas"], "magFlux": nxt["mf"], "Bxyz": nxt["B"], "dGas": d[0], "dmagFlux": d[1], "doGas": d[2],
            "domagFlux": d[3]}


def work(case):
    """Bytes: state in and out and the metric, each once per step (27 + 79
    values per cell, 24 more of FP64 background field where there is one), and
    the output that crosses to the host. Operations: the step's arithmetic per
    cell-update, about 3000."""
    n = _n(case)
    cells = n[0] * n[1] * n[2]
    w = 4 if case["form"] == "fp32" else 8
    per = 106 * w + (192 if case["problem"] in ("dipole", "lfm") else 0)
    box = (n[0] + 8) * (n[1] + 8) * (n[2] + 8)
    steps = case["steps"]
    if case["kind"] == "sweep":
        # forward, and backward with the metric and both states once more
        return {"bytes": cells * steps * 2.0 * per, "flops": cells * steps * 9000.0}
    if case["kind"] == "adjoint":
        return {"bytes": cells * (2.0 * per + 27 * w), "flops": cells * 9000.0}
    out = {"forward": 11, "dropin": 24}[case["kind"]] * box * 8.0
    return {"bytes": cells * steps * float(per) + out, "flops": cells * steps * 3000.0}


def tolerance(case):
    # rel: 2-norm; max: the largest difference over the rms. Differences from
    # exact() measured over the listed cases, times about four: FP64 1e-12 (the
    # vortex after 100 steps; its shocks amplify rounding), FP32 2e-7 on the
    # blast; next to the polar axis of the dipole's grid FP32 is 1e-5 off in the
    # transverse momenta. Gradients 3e-13
    if case["kind"] in ("sweep", "adjoint"):
        return {"rel": 1e-10, "max": 1e-6}
    if case["form"] == "fp32":
        return {"rel": 1e-5, "max": 1e-3} if case["problem"] in ("dipole", "lfm") else {"rel": 1e-6, "max": 1e-4}
    return {"rel": 5e-12, "max": 1e-9}


# ----------------------------------------------------------------- 64-bit values
# The step in plain torch on the ghosted box (every field (..., Nk+9, Nj+9,
# Ni+9), cell fields without their last slots), periodic boundaries.
_W8 = [q / 840.0 for q in (-3, 29, -139, 533, 533, -139, 29, -3)]
_UP = [q / 420.0 for q in (-3, 25, -101, 319, 214, -38, 4)]


class _Exact:
    def __init__(self, case, xyz, gamma=5.0 / 3.0):
        self.n = _n(case)
        self.up7 = case["recon"] == "7up"
        self.lfm = case["option"] != "nolfmlim"
        self.d25 = case["problem"] == "ot" and case["nk"] == 1
        self.gm1, self.gamma, self.dev = gamma - 1, gamma, "cuda" if torch.cuda.is_available() else "cpu"
        x = torch.as_tensor(xyz, dtype=torch.float64, device=self.dev)
        self.size = tuple(x.shape[1:])
        self.all = [(0, s - 1) for s in self.size[::-1]]        # cell ranges i, j, k
        self.metric(x)
        self.maps()

    # windows: ranges r = [(i0, i1), (j0, j1), (k0, k1)), half open, shifted by n along d
    def w(self, a, r, d=0, n=0, d2=0, n2=0):
        s = []
        for q in (2, 1, 0):
            o = (n if q == d else 0) + (n2 if q == d2 else 0)
            s.append(slice(r[q][0] + o, r[q][1] + o))
        return a[(Ellipsis, *s)]

    def put(self, a, r):
        out = torch.zeros(a.shape[:-3] + self.size, dtype=a.dtype, device=a.device)
        s = tuple(slice(*r[q]) for q in (2, 1, 0))
        out[(Ellipsis, *s)] = a
        return out

    def metric(self, x):
        S, n = self.size[::-1], self.n
        gl, gw = np.polynomial.legendre.leggauss(12)
        full = [(0, s) for s in S]
        self.area, self.cen, self.tri = [], [], []
        for d in range(3):
            a1, a2 = (d + 1) % 3, (d + 2) % 3
            r = [list(q) for q in full]
            r[a1][1] -= 1
            r[a2][1] -= 1
            f0, f1, f2, f3 = self.w(x, r), self.w(x, r, a1, 1), self.w(x, r, a2, 1), self.w(x, r, a1, 1, a2, 1)
            e1, e2, e3 = f1 - f0, f2 - f0, f3 + f0 - f2 - f1
            A, m = 0, 0
            for i in range(12):
                for j in range(12):
                    u, v = 0.5 * (1 + gl[i]), 0.5 * (1 + gl[j])
                    c = torch.linalg.vector_norm(torch.linalg.cross(e1 + e3 * v, e2 + e3 * u, dim=0), dim=0)
                    c = c * (0.25 * gw[i] * gw[j])
                    A = A + c
                    m = m + c * (f0 + e1 * u + e2 * v + e3 * (u * v))
            self.area.append(self.put(A, r))
            self.cen.append(self.put(m / A, r))
            t1, t2 = 0.5 * (f3 - f2 + f1 - f0), 0.5 * (f3 - f1 + f2 - f0)
            def unit(q):
                return q / torch.linalg.vector_norm(q, dim=0)
            nn, t2 = unit(torch.linalg.cross(t1, t2, dim=0)), unit(t2)
            self.tri.append([self.put(q, r) for q in (nn, unit(torch.linalg.cross(t2, nn, dim=0)), t2)])
        # volume and barycentre: two Gauss points per direction integrate the trilinear map exactly
        r = [(0, s - 1) for s in S]
        V, xc = 0, 0
        g2 = 1 / math.sqrt(3.0)
        corner = [[[x[(slice(None), slice(k, S[2] - 1 + k), slice(j, S[1] - 1 + j), slice(i, S[0] - 1 + i))]
                    for i in (0, 1)] for j in (0, 1)] for k in (0, 1)]
        for p in range(8):
            t = [0.5 * (1 + (g2 if p >> q & 1 else -g2)) for q in range(3)]
            pos, J = 0, [0, 0, 0]
            for k in (0, 1):
                for j in (0, 1):
                    for i in (0, 1):
                        f = [t[q] if o else 1 - t[q] for q, o in enumerate((i, j, k))]
                        g = [1.0 if o else -1.0 for o in (i, j, k)]
                        c = corner[k][j][i]
                        pos = pos + c * (f[0] * f[1] * f[2])
                        J[0] = J[0] + c * (g[0] * f[1] * f[2])
                        J[1] = J[1] + c * (f[0] * g[1] * f[2])
                        J[2] = J[2] + c * (f[0] * f[1] * g[2])
            dJ = (torch.linalg.cross(J[0], J[1], dim=0) * J[2]).sum(0).abs() / 8
            V, xc = V + dJ, xc + dJ * pos
        self.vol, xcc = self.put(V, r), self.put(xc / V, r)
        self.xcc = xcc
        self.dl = None
        for d in range(3):
            q = self.w(self.vol, r) / torch.maximum(self.w(self.area[d], r, d, 1), self.w(self.area[d], r))
            self.dl = q if self.dl is None else torch.minimum(self.dl, q)
        # centroid of the lower / upper face minus that of the cell
        self.off = [[self.w(self.cen[d], r, d, o) - self.w(xcc, r) for o in (0, 1)] for d in range(3)]
        # edges: length, the two tangents and the face normals seen from them, on the active edges
        ar = [(NG, NG + q + 1) for q in n]
        self.edge, self.et, self.eb = [], [], []
        for d in range(3):
            p, q = (1, 2) if d == 0 else (2, 0) if d == 1 else (0, 1)
            c = (2, 0, 1)[d]                                   # the direction eAvg runs along
            de = self.w(x, ar, d, 1) - self.w(x, ar)
            av = 0.5 * (self.w(x, ar, c, 1) - self.w(x, ar, c, -1) + self.w(x, ar, d, 1, c, 1) -
                        self.w(x, ar, d, 1, c, -1))
            L = torch.linalg.vector_norm(de, dim=0)
            e = de / L
            t1 = torch.linalg.cross(av, e, dim=0)
            t1 = t1 / torch.linalg.vector_norm(t1, dim=0)
            t2 = torch.linalg.cross(e, t1, dim=0)
            t2 = t2 / torch.linalg.vector_norm(t2, dim=0)
            self.edge.append(L)
            self.et.append((t1, t2))
            nb = []
            for fd, sd in ((p, q), (q, p)):                    # faces of direction fd, stencil along sd
                w6 = [0, 1 / 60, -8 / 60, 37 / 60, 37 / 60, -8 / 60, 1 / 60, 0]
                ne = sum(w6[m] * self.w(self.tri[fd][0], ar, sd, m - 4) * self.w(self.area[fd], ar, sd, m - 4)
                         for m in range(1, 7))
                fa = sum(w6[m] * self.w(self.area[fd], ar, sd, m - 4) for m in range(1, 7))
                ne = ne / fa
                a, b = (ne * t1).sum(0), (ne * t2).sum(0)
                s = torch.sqrt(a * a + b * b)
                s = torch.where(s <= 1e-12, torch.ones_like(s), s)
                nb += [a / s, b / s]
            self.eb.append(nb)

    def maps(self):
        """Periodic images on the ghosted box, per kind of value."""
        S, n = self.size, self.n
        self.src = {}
        for comp in (-1, 0, 1, 2):
            ax = []
            for q in range(3):
                x = np.arange(S[2 - q])
                f = 1 if comp == q else 0                      # the upper face of the last cell is its own
                hi = (x >= NG + n[q] + f) & (x <= NG + n[q] + 3 + f)
                ax.append(np.where(x < NG, NG + (x - NG) % n[q], np.where(hi, NG + f + (x - NG - f) % n[q], x)))
            if comp == -1:
                for q in range(3):
                    ax[q][-1] = S[2 - q] - 1
            full = (ax[2][:, None, None] * S[1] + ax[1][None, :, None]) * S[2] + ax[0][None, None, :]
            if comp == -1:
                own = np.arange(full.size).reshape(full.shape)
                out = np.zeros(full.shape, bool)
                out[-1], out[:, -1], out[:, :, -1] = True, True, True
                full = np.where(out, own, full)
            self.src[comp] = torch.as_tensor(full.reshape(-1), device=self.dev)

    def fill(self, gas, mf):
        flat = lambda a, c: a.reshape(*a.shape[:-3], -1)[..., self.src[c]].reshape(a.shape)  # noqa: E731
        return flat(gas, -1), torch.stack([flat(mf[d], d) for d in range(3)])

    def field(self, mf):
        r = self.all
        b = 0
        for d in range(3):
            b = b + self.w(mf[d], r, d, 1) * self.off[d][1] - self.w(mf[d], r) * self.off[d][0]
        return self.put(b / self.w(self.vol, r), r)

    def prim(self, u):
        v = u[1:4] / u[0]
        return torch.cat([u[:1], v, (self.gm1 * (u[4] - 0.5 * u[0] * (v * v).sum(0)))[None].clamp_min(1e-12)])

    @staticmethod
    def limit(v0, v1, v2, q):
        """The left state between cells v1 and v2."""
        q = torch.maximum(torch.minimum(v1, v2), torch.minimum(q, torch.maximum(v1, v2)))
        d0, d1 = 0.75 * (v1 - v0), 0.75 * (v2 - v1)
        one = torch.ones_like(d0)
        s0, s1 = torch.copysign(one, d0), torch.copysign(one, d1)
        return q - s1 * torch.clamp_min((q - v1).abs() - (s0 + s1).abs() * d0.abs(), 0.0)

    def lr(self, Q, L, Vi, r, d):
        """Left and right states on the faces r of direction d: Q the weighted stencil, L the limiter values."""
        v = [self.w(L, r, d, m) for m in (-2, -1, 0, 1)]
        if self.up7:
            a = sum(_UP[m] * self.w(Q, r, d, m - 4) for m in range(7)) / Vi
            b = sum(_UP[m] * self.w(Q, r, d, 3 - m) for m in range(7)) / Vi
        else:
            a = b = sum(_W8[m] * self.w(Q, r, d, m - 4) for m in range(8)) / Vi
        return self.limit(v[0], v[1], v[2], a), self.limit(v[3], v[2], v[1], b)

    def mid(self, a, r, d):
        return sum(_W8[m] * self.w(a, r, d, m - 4) for m in range(8))

    def step(self, cur, old, dt, odt, want_dt=False):
        gas, mf, B = cur
        ogas, omf = old[0], old[1]
        r, n, gm1 = self.all, self.n, self.gm1
        g, og = self.w(gas, r), self.w(ogas, r)
        W, oW = self.prim(g), self.prim(og)
        H = W + 0.5 * dt * ((W - oW) / odt)
        H = torch.cat([H[:1].clamp_min(1e-12), H[1:4], H[4:].clamp_min(1e-12)])
        hm = mf + 0.5 * dt * ((mf - omf) / odt)
        hB = self.field(hm)
        vol = self.w(self.vol, r)
        half, now = self.put(H, r), self.put(W, r)
        QW, QB = self.put(vol * H, r), self.vol * hB
        Wl, Bl = (now, B) if self.lfm else (half, hB)
        # edge EMFs
        E = []
        for d in range(3):
            d1, d2 = (d + 1) % 3, (d + 2) % 3
            re = [(NG, NG + n[q] + (0 if q == d else 1)) for q in range(3)]
            cut = lambda a: a[(Ellipsis, *(slice(0, re[q][1] - re[q][0]) for q in (2, 1, 0)))]  # noqa: E731
            rf = [(0, self.size[2 - q] - 1) for q in range(3)]
            rf[d1] = re[d1]
            Vf = self.mid(QW[1:4], rf, d1) / self.mid(self.vol, rf, d1)
            AVf = self.put(self.w(self.area[d1], rf) * Vf, rf)
            ab = []
            for fd, sd in ((d1, d2), (d2, d1)):
                A = self.mid(self.area[fd], re, sd)
                safe = self.area[fd].clamp_min(1e-12)
                Lm = (mf[fd] if self.lfm else hm[fd]) / safe
                L, R = self.lr(hm[fd], Lm, A, re, sd)
                ab.append((A, L, R))
            (A1, L1, R1), (A2, L2, R2) = ab
            V = self.mid(AVf, re, d2) / A1
            t1, t2 = cut(self.et[d][0]), cut(self.et[d][1])
            v1, v2 = (V * t1).sum(0), (V * t2).sum(0)
            xi, yi, xj, yj = [cut(q) for q in self.eb[d]]
            det = 1 / (xi * yj - xj * yi)
            c1, c2 = 0.5 * (L1 + R1), 0.5 * (L2 + R2)
            Jd = (R2 - L2) - (R1 - L1)
            b1, b2 = det * (yj * c1 - yi * c2), det * (xi * c2 - xj * c1)
            e1, e2 = (q for q in range(3) if q != d)
            D = 0.25 * sum(self.w(half[0], re, e1, -i, e2, -j) for i in (0, 1) for j in (0, 1))
            def root(q):  # a zero derivative at zero
                return torch.where(q > 0, torch.sqrt(torch.where(q > 0, q, torch.ones_like(q))), torch.zeros_like(q))
            vD = root(v1 * v1 + v2 * v2) + root(b1 * b1 + b2 * b2) / torch.sqrt(D)
            L = cut(self.edge[d])
            vD = torch.minimum(vD, 0.3 * L / dt)
            E.append(self.put((-(v1 * b2 - v2 * b1) + 0.5 * vD * Jd) * L, re))
        # face fluxes
        dU, dM = 0, 0
        act = [(NG, NG + q) for q in n]
        for d in range(3):
            rf = [(NG, NG + n[q] + (1 if q == d else 0)) for q in range(3)]
            if d == 2 and self.d25:
                continue
            N, T1, T2 = [self.w(q, rf) for q in self.tri[d]]
            fa = self.w(self.area[d], rf)
            Vi = self.mid(self.vol, rf, d)
            Bn = self.w(hm[d], rf) / fa
            sides = list(zip((-1.0, 1.0), self.lr(QW, Wl, Vi, rf, d), self.lr(QB, Bl, Vi, rf, d)))
            F, M, va, dW = 0, 0, 0, 0
            for s, w, b in sides:
                rho, v, p = w[0], w[1:4], w[4]
                pb = 0.5 * (b * b).sum(0)
                va2 = 2 * pb / rho
                vn, vt1, vt2 = (N * v).sum(0), (T1 * v).sum(0), (T2 * v).sum(0)
                half_ = 0.5 * torch.erfc(s * vn / torch.sqrt(2 * p / rho + va2))
                M = M + half_ * (pb * N - b * Bn)
                va = va + 0.5 * torch.where(va2 > 0, torch.sqrt(torch.where(va2 > 0, va2, torch.ones_like(va2))),
                                            torch.zeros_like(va2))
                lam = rho / (2 * p)
                v0 = 0.5 * torch.erfc(s * torch.sqrt(lam) * vn)
                v1 = vn * v0 - 0.5 * s * torch.exp(-lam * vn * vn) / torch.sqrt(PI * lam)
                e = 0.5 * rho * (v * v).sum(0) + p / gm1
                mom = N * (rho * vn * v1 + p * v0) + T1 * (rho * vt1 * v1) + T2 * (rho * vt2 * v1)
                F = F + torch.cat([(rho * v1)[None], mom, ((e + 0.5 * p) * v1 + 0.5 * p * v0 * vn)[None]])
                dW = dW + s * torch.cat([rho[None], rho * v, e[None]])
            F, M = self.put(fa * (F - 0.25 * va * dW), rf), self.put(fa * M, rf)
            dU = dU + self.w(F, act) - self.w(F, act, d, 1)
            dM = dM + self.w(M, act) - self.w(M, act, d, 1)
        # update
        rE = [(NG, NG + q + 1) for q in n]
        def curl(a, da, b, db):
            return self.w(E[a], rE, da, 1) - self.w(E[a], rE) - self.w(E[b], rE, db, 1) + self.w(E[b], rE)
        rot = torch.stack([curl(2, 1, 1, 2), curl(0, 2, 2, 0), curl(1, 0, 0, 1)])
        mfn = mf - dt * self.put(rot, rE)
        vol = self.w(self.vol, act)
        U = self.w(gas, act) + dt * dU / vol
        rho = U[0].clamp_min(1e-12)
        p = (gm1 * (U[4] - 0.5 * (U[1:4] ** 2).sum(0) / rho)).clamp_min(1e-12)
        mom = U[1:4] + dt * dM / vol
        new = torch.cat([rho[None], mom, (0.5 * (mom ** 2).sum(0) / rho + p / gm1)[None]])
        keep = gas - self.put(self.w(gas, act), act)
        gasn = keep + self.put(new, act)
        if want_dt:  # CalcDT comes before the boundaries: its ghost layer holds the step's start
            dt = self.cfl(gasn, self.field(mfn))
        gasn, mfn = self.fill(gasn, mfn)
        return (gasn, mfn, self.field(mfn)) + ((dt,) if want_dt else ())

    def cfl(self, gas, B):
        u, b = self.w(gas, self.all), self.w(B, self.all)
        v = u[1:4] / u[0]
        p = self.gm1 * (u[4] - 0.5 * u[0] * (v * v).sum(0))
        c = torch.sqrt((v * v).sum(0)) + torch.sqrt(self.gamma * p / u[0] + (b * b).sum(0) / u[0])
        q = 0.3 * self.dl / c
        s = tuple(slice(NG - 1, NG + m + 1) for m in self.n[::-1])
        return float(q[s].min())

    def blast(self, x0, y0, z0, pRat, rC):
        """Gas averaged over the cells by 12 Gauss points per direction (only the
        cells that the sphere's surface can cut need it), uniform field."""
        r, S = self.all, self.size[::-1]
        x = self.x
        c = x.new_tensor([x0, y0, z0]).reshape(3, 1, 1, 1)
        corner = [x[(slice(None), slice(k, S[2] - 1 + k), slice(j, S[1] - 1 + j), slice(i, S[0] - 1 + i))]
                  for k in (0, 1) for j in (0, 1) for i in (0, 1)]
        mid = sum(corner) / 8
        reach = torch.stack([torch.linalg.vector_norm(q - mid, dim=0) for q in corner]).amax(0)
        R = torch.linalg.vector_norm(mid - c, dim=0)
        p = 0.1 + (R <= rC) * (0.1 * (pRat - 1.0) * torch.ones_like(R))
        cutm = (R - rC).abs() <= 1.01 * reach
        cc = torch.stack([q[:, cutm] for q in corner])           # (8, 3, m)
        gl, gw = np.polynomial.legendre.leggauss(12)
        tot = 0
        for i in range(12):
            for j in range(12):
                f, J = [], []
                u, v = 0.5 * (1 + gl[i]), 0.5 * (1 + gl[j])
                w = torch.as_tensor(0.5 * (1 + gl), device=self.dev)
                k0 = [cc[q] * ((u if q & 1 else 1 - u) * (v if q & 2 else 1 - v)) for q in range(8)]
                lo, hi = sum(k0[:4]), sum(k0[4:])
                pos = lo[None] * (1 - w)[:, None, None] + hi[None] * w[:, None, None]
                du = [cc[q] * ((1 if q & 1 else -1) * (v if q & 2 else 1 - v)) for q in range(8)]
                dv = [cc[q] * ((u if q & 1 else 1 - u) * (1 if q & 2 else -1)) for q in range(8)]
                Ju = sum(du[:4])[None] * (1 - w)[:, None, None] + sum(du[4:])[None] * w[:, None, None]
                Jv = sum(dv[:4])[None] * (1 - w)[:, None, None] + sum(dv[4:])[None] * w[:, None, None]
                Jw = (hi - lo)[None].expand_as(Ju)
                dJ = (torch.linalg.cross(Ju, Jv, dim=1) * Jw).sum(1).abs()
                inside = torch.linalg.vector_norm(pos - c.reshape(1, 3, 1), dim=1) <= rC
                ww = torch.as_tensor(gw, device=self.dev)[:, None] * (gw[i] * gw[j] / 8)
                tot = tot + (ww * dJ * (0.1 + inside * (0.1 * (pRat - 1.0) * torch.ones_like(dJ)))).sum(0)
        vol = self.w(self.vol, r)
        p[cutm] = tot / vol[cutm]
        gas = torch.zeros((5,) + self.size, dtype=torch.float64, device=self.dev)
        gas[(0, *(slice(0, s - 1) for s in self.size))] = 1.0
        gas[(4, *(slice(0, s - 1) for s in self.size))] = p / self.gm1
        b = float(np.float32(math.sqrt(2.0)))
        mf = []
        for d in range(3):                                       # uniform field: B . (half the diagonals' cross product)
            a1, a2 = (d + 1) % 3, (d + 2) % 3
            rr = [[0, s] for s in S]
            rr[a1][1] -= 1
            rr[a2][1] -= 1
            f0, f1, f2, f3 = self.w(x, rr), self.w(x, rr, a1, 1), self.w(x, rr, a2, 1), self.w(x, rr, a1, 1, a2, 1)
            A = 0.5 * torch.linalg.cross(f3 - f0, f2 - f1, dim=0)
            mf.append(self.put((A[0] + A[1]) / b, rr))
        return self.fill(gas, torch.stack(mf))


def _start(case, seed, ex, xyz):
    if case["problem"] == "ot":
        gas, mf = _vortex(case, seed)
        gas, mf = torch.as_tensor(gas, device=ex.dev), torch.as_tensor(mf, device=ex.dev)
        return ex.put(gas, ex.all), mf
    ex.x = torch.as_tensor(xyz, dtype=torch.float64, device=ex.dev)
    return ex.blast(**_blast(seed))


def exact(case, seed):
    """None for the problems whose boundaries (sphere, wind, ionosphere, rings)
    and options (Boris, AB3) the plain step here does not have."""
    n = _n(case)
    if case["problem"] not in ("ot", "blast") or case["option"] in ("boris", "ab3"):
        return None
    if n[0] * n[1] * n[2] * case["steps"] > 8e7:
        return None
    xyz = _corners(case)
    ex = _Exact(case, xyz)
    gas, mf = _start(case, seed, ex, xyz)
    cells = lambda a: a[..., :-1, :-1, :-1]  # noqa: E731
    dt = ex.cfl(gas, ex.field(mf))
    if case["kind"] in ("forward", "dropin"):
        cur = (gas, mf, ex.field(mf))
        old, odt, t = cur, dt, 0.0
        for _ in range(case["steps"]):
            *new, dtn = ex.step(cur, old, dt, odt, want_dt=True)
            old, cur, odt, t, dt = cur, new, dt, t + dt, dtn
        out = {"Gas": cells(cur[0]), "magFlux": cur[1]}
        if case["kind"] == "forward":
            out["Bxyz"] = cells(cur[2])
        return {k: v.cpu().numpy() for k, v in out.items()} | {"dt": dt, "time": t, "otime": t - odt,
                                                               "ts": case["steps"]}
    dtype = torch.float32 if case["form"] == "fp32" else torch.float64
    dt = 0.5 * dt
    # the same rounded start that the form gets
    ngas, nmf = _noises(n, seed, dtype)
    gas = (gas.to(dtype) + 1e-3 * (gas.to(dtype) + _still(dtype, ex.dev)) * ngas).double()
    mf = (mf.to(dtype) + 1e-3 * torch.stack(ex.area).to(dtype) * nmf).double()
    if case["kind"] == "adjoint":
        old = (gas, mf, ex.field(mf))
        cur = ex.step(old, old, dt, dt)
        cur = tuple(q.to(dtype).double() for q in cur)
        leaves = [q.detach().requires_grad_(True) for q in (cur[0], cur[1], old[0], old[1])]
        c, o = (leaves[0], leaves[1], ex.field(leaves[1])), (leaves[2], leaves[3], ex.field(leaves[3]))
        out = ex.step(c, o, dt, dt)
        dn = [q.double() for q in _noises(n, seed + 11, dtype)]
        d = torch.autograd.grad([out[0], out[1]], leaves, dn)
        return {"Gas": out[0].detach(), "magFlux": out[1].detach(), "Bxyz": out[2].detach(), "dGas": d[0],
                "dmagFlux": d[1], "doGas": d[2], "domagFlux": d[3]}
    G0, M0 = gas.requires_grad_(True), mf.requires_grad_(True)
    from torch.utils.checkpoint import checkpoint
    cur = (G0, M0, ex.field(M0))
    old = cur
    for _ in range(case["steps"]):
        new = checkpoint(lambda a, b, c, d, e, f: ex.step((a, b, c), (d, e, f), dt, dt), *cur, *old, use_reentrant=False)
        old, cur = cur, new
    b = cells(cur[2])
    xc = cells(ex.xcc)
    act = tuple(slice(NG, NG + q) for q in n[::-1])
    m = ((xc >= 0.6) & (xc <= 0.8)).all(0)[act]
    loss = ((b * b).sum(0)[act] * m).sum()
    d = torch.autograd.grad(loss, [G0, M0])
    return {"loss": float(loss.detach()), "dGas": d[0], "dmagFlux": d[1]}
