"""Performance cases of the multislice engine.

Each case is a piece of work a simulation program gives the engine, through
the public calls of ``ManagedMultisliceSimulation``:

``steps``      the interactive loop: initial wave, one call per slice, exit wave
``structure``  a new structure through the whole run: atoms in, binning,
               potentials, slices, then the exit wave or the CTF image
``run``        slices over the resident potential stack, exit wave out
``raster``     a STEM probe raster over the resident stack, detector signals
``phonon``     a frozen-phonon series: mean diffraction and image
``forward``    one evaluation of a focal-series fit after the atoms moved
``grad``       the same with its gradient (atom positions and/or potentials)
``fd``         a finite-difference run over its resident potential planes
``images``     a defocus sweep of one exit wave

Specimens are seeded: amorphous carbon as a jittered lattice at 0.1 atoms/A^3
and crystals with thermal-sized displacements.  ``exact`` restates the path in
FP64 with torch; the FP32 decisions that define the problem (z-bins, cut-offs,
apertures, band limit) and the FP32 set-up scalars are taken as the engine's
documentation states them.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

import cudamultislice_b200 as ms

F = np.float32
DATA = os.path.join(os.path.dirname(os.path.abspath(ms.__file__)), "data", "fparams.dat")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call sequence: a preview grid stepped slice by slice
        dict(name="steps_64", kind="steps", specimen="srtio3", nx=64, ny=64, sx=7.81, depth=12.0, dz=1.9525, kV=200.0),
        # SrTiO3 4 x 4 x 20 cells on 256^2, 200 kV: a small structure to its image
        dict(name="structure_256", kind="structure", specimen="srtio3", nx=256, ny=256, sx=15.62, depth=78.1, dz=1.9525,
             kV=200.0, image=True),
        # the amorphous slab at 1024^2 from host atoms to host exit wave
        dict(name="structure_1024", kind="structure", specimen="carbon", nx=1024, ny=1024, sx=50.0, depth=200.0, dz=2.0,
             kV=300.0, image=False),
        # a grid that is no power of two (per-operation path)
        dict(name="structure_600x450", kind="structure", specimen="silicon", nx=600, ny=450, sx=43.4, depth=60.0,
             dz=1.92, kV=200.0, image=False),
        # repeated slice loops over a resident stack, the headline workload
        dict(name="run_1024", kind="run", specimen="carbon", nx=1024, ny=1024, sx=50.0, depth=196.0, dz=2.0, kV=300.0),
        # a strip: rows and columns of different length
        dict(name="run_512x256", kind="run", specimen="gan", nx=512, ny=256, sx=36.0, depth=80.0, dz=1.5945, kV=300.0),
        # the largest grid
        dict(name="run_4096", kind="run", specimen="carbon", nx=4096, ny=4096, sx=50.0, depth=44.0, dz=2.0, kV=300.0),
        # HAADF raster on 1024^2, probes per launch left to the engine
        dict(name="raster_1024", kind="raster", specimen="gan", nx=1024, ny=1024, sx=54.0, depth=64.0, dz=1.5945,
             kV=300.0, probes=128, batch=0),
        # thermal configurations of silicon on 512^2
        dict(name="phonon_512", kind="phonon", specimen="silicon", nx=512, ny=512, sx=32.6, depth=96.0, dz=1.92, kV=200.0,
             configs=16, batch=16),
        # one step of a position refinement: forward and adjoint from moved atoms
        dict(name="grad_512", kind="grad", specimen="srtio3", nx=512, ny=512, sx=15.62, depth=97.6, dz=1.9525, kV=200.0,
             images=8, want_v=False),
        # finite-difference steps of a quarter slice
        dict(name="fd_512", kind="fd", specimen="carbon", nx=512, ny=512, sx=25.0, depth=60.0, dz=2.0, kV=300.0, steps=96,
             fd_dz=0.5),
        # defocus sweep of one exit wave
        dict(name="images_1024", kind="images", specimen="carbon", nx=1024, ny=1024, sx=50.0, depth=10.0, dz=2.0, kV=300.0,
             images=8),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _budget(c):
    """Slices x instances x pixels: bounded by the listed cases of each kind."""
    inst = {"raster": c.get("probes", 1), "phonon": c.get("configs", 1), "grad": 3}.get(c["kind"], 1)
    return inst * math.ceil((c["depth"] + 4.0) / c["dz"]) * c["nx"] * c["ny"]


def draw(rng):
    kind = rng.choice(["steps", "structure", "structure", "run", "run", "raster", "phonon", "grad", "forward", "fd", "images"])
    specimen = rng.choice(["carbon", "srtio3", "silicon", "gan"])
    top = {"steps": 10, "structure": 11, "run": 12, "raster": 10, "phonon": 9, "grad": 9, "forward": 10, "fd": 10, "images": 11}[kind]
    nx = 2 ** rng.randint(6, top)
    ny = nx if rng.random() < 0.6 else 2 ** min(top, max(6, int(math.log2(nx)) + rng.choice([-1, 1])))
    if kind in ("steps", "structure", "run", "fd", "images") and rng.random() < 0.25:
        # any even or odd size: the general path
        nx, ny = (int(_log_uniform(rng, 70, 1000)) for _ in range(2))
    c = dict(kind=kind, specimen=specimen, nx=nx, ny=ny, sx=round(nx * _log_uniform(rng, 0.03, 0.1), 2),
             depth=round(_log_uniform(rng, 8.0, 200.0), 1), dz=round(rng.uniform(1.0, 2.5), 3),
             kV=rng.choice([80.0, 200.0, 300.0]))
    if kind == "structure":
        c["image"] = rng.random() < 0.4
    if kind == "raster":
        c.update(probes=int(_log_uniform(rng, 3, 128)), batch=rng.choice([0, 7, 16, 32]))
    if kind == "phonon":
        c.update(configs=int(_log_uniform(rng, 2, 24)), batch=rng.choice([3, 8, 16]))
    if kind in ("grad", "forward", "images"):
        c.update(images=rng.randint(1, 8))
    if kind == "grad":
        c["want_v"] = rng.random() < 0.5
    if kind == "fd":
        c.update(steps=int(_log_uniform(rng, 9, 130)), fd_dz=0.5)
    # no more than the largest listed case's work, nor its atoms and planes
    cap = {"steps": 3e7, "structure": 1.0e8, "run": 1.5e8, "raster": 3e9, "phonon": 2.2e8, "grad": 4e7, "forward": 4e7,
           "fd": 1e9, "images": 2e7}[kind]
    while _budget(c) > cap and c["depth"] > 8.0:
        c["depth"] = round(max(8.0, 0.8 * c["depth"]), 1)
    if kind == "raster":
        c["probes"] = max(2, min(c["probes"], int(c["probes"] * cap / _budget(c))))
    if kind == "fd":
        c["steps"] = max(9, min(c["steps"], int(3.0e7 / (nx * ny))))
        c["depth"] = round(max(8.0, c["steps"] * c["fd_dz"]), 1)
    sy = c["sx"] * ny / nx
    c["depth"] = round(min(c["depth"], max(8.0, 5.0e5 / (c["sx"] * sy))), 1)
    return c


# ---------------------------------------------------------------------------
# specimens
# ---------------------------------------------------------------------------
_ZINC = [(0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0)]
_CELLS = {
    "srtio3": (3.905, [(0, 0, 0), (.5, .5, .5), (.5, .5, 0), (.5, 0, .5), (0, .5, .5)], [38, 22, 8, 8, 8]),
    "silicon": (5.431, _ZINC + [(a + .25, b + .25, c + .25) for a, b, c in _ZINC], [14] * 8),
    "gan": (4.50, _ZINC + [(a + .25, b + .25, c + .25) for a, b, c in _ZINC], [31] * 4 + [7] * 4),
    "carbon": (2.1544, [(0, 0, 0)], [6]),
}


def _atoms(case, rng):
    a, basis, Zc = _CELLS[case["specimen"]]
    sy = case["sx"] * case["ny"] / case["nx"]
    n = [max(1, int(round(s / a))) for s in (case["sx"], sy, case["depth"])]
    g = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 1, 3)
    pos = ((g + np.asarray(basis)[None]) * a).reshape(-1, 3)
    jitter = rng.uniform(-0.45, 0.45, pos.shape) if case["specimen"] == "carbon" else rng.normal(0.0, 0.08, pos.shape)
    pos = (pos + jitter).astype(F)
    Z = np.tile(np.asarray(Zc, np.int32), g.shape[0])
    return Z, *(np.ascontiguousarray(pos[:, k]) for k in range(3))


def _inputs(case, seed):
    rng = np.random.default_rng([seed, case["nx"], case["ny"]])
    d = {"atoms": _atoms(case, rng), "rng": rng}
    nx, ny = case["nx"], case["ny"]
    if case["kind"] == "raster":
        d["px"] = rng.integers(nx // 8, nx - nx // 8, case["probes"]).astype(np.int32)
        d["py"] = rng.integers(ny // 8, ny - ny // 8, case["probes"]).astype(np.int32)
    if "images" in case:
        d["defoci"] = np.linspace(-800.0, 600.0, case["images"]).astype(F)
    if case["kind"] in ("grad", "forward"):
        d["targets"] = (1.0 + 0.2 * rng.standard_normal((case["images"], ny, nx))).astype(F)
    return d


def _micro(case):
    stem = case["kind"] == "raster"
    return dict(kV=case["kV"], df=0.0 if stem else -500.0, Cs=0.0 if stem else 1.2e7, beta=0.1, delta=30.0,
                ap=25.0 if stem else 20.0, ps=case["sx"] / case["nx"])


# ---------------------------------------------------------------------------
# the engine's side
# ---------------------------------------------------------------------------
def prepare(case, seed):
    d, m = _inputs(case, seed), _micro(case)
    nx, ny, kind = case["nx"], case["ny"], case["kind"]
    sim = ms.ManagedMultisliceSimulation()
    sim.SetAtoms(*d["atoms"])
    sim.UploadBinnedAtoms()
    sim.GetParameterisation(DATA)
    sim.ApplyMicroscopeParameters(m["kV"], m["df"], 0.0, 0.0, m["Cs"], m["beta"], m["delta"], m["ap"])
    size = (sim.GetSizeX(), sim.GetSizeY(), sim.GetSizeZ())
    if kind == "raster":
        sim.STEMSetCalculationVariables(m["ps"], m["df"], nx, ny, *size)
    else:
        sim.SetCalculationVariables(m["ps"], m["df"], nx, ny, *size, 2.0, 2.0)
    sim.PreCalculateFrequencies()
    if kind == "fd":
        sim.SetFDdz(case["fd_dz"])
    sim.InitialiseWavefunctions(case["dz"])
    if kind in ("run", "raster"):
        sim.BuildPotentialStack()
    if kind == "images":
        sim.RunConventional()
    d.update(sim=sim, case=case, seed=seed, slices=sim.GetSlices(True),
             wave=torch.zeros((ny, nx), dtype=torch.complex64).pin_memory().numpy())
    return d


def run(state):
    sim, case = state["sim"], state["case"]
    kind = case["kind"]
    if kind == "steps":
        sim.InitialiseWavefunctions(case["dz"])
        for i in range(1, state["slices"] + 1):
            sim.MultisliceStepConventional(i)
        return {"wave": sim.ExitWave(state["wave"])}
    if kind == "structure":
        sim.SetAtoms(*state["atoms"])
        sim.UploadBinnedAtoms()
        sim.RunConventional()
        if case["image"]:
            sim.SimulateImage()
            return {"image": sim.Image()}
        return {"wave": sim.ExitWave(state["wave"])}
    if kind == "run":
        sim.RunConventional()
        return {"wave": sim.ExitWave(state["wave"])}
    if kind == "raster":
        # (detector sums of single-precision waves: compared as such)
        return {"signal": sim.StemRaster(state["px"], state["py"], 70.0, 200.0, batch=case["batch"]).astype(F)}
    if kind == "phonon":
        diff, image = sim.FrozenPhonon(state["seed"] + 1, 0, case["configs"], 0.076, batch=case["batch"])
        return {"diffraction": diff, "image": image}
    if kind in ("grad", "forward"):
        sim.SetAtoms(*state["atoms"])
        sim.UploadBinnedAtoms()
        if kind == "forward":
            loss, images = sim.FocalSeries(state["defoci"], state["targets"], state["slices"], images=True)
            return {"loss": loss, "images": images}
        loss, gv, gxy = sim.FocalSeriesGrad(state["defoci"], state["targets"], state["slices"], want_v=case["want_v"])
        out = {"loss": loss, "dxy": gxy.astype(F)}  # (sums of single-precision terms)
        if case["want_v"]:
            out["dv"] = gv
        return out
    if kind == "fd":
        sim.InitialiseWavefunctions(case["dz"])
        sim.RunFD(case["steps"])
        return {"wave": sim.ExitWave(state["wave"])}
    if kind == "images":
        return {"images": sim.SimulateImageSeries(state["defoci"])}
    raise ValueError(kind)


def work(case):
    """Inputs read and results written once; transforms at 5 N log2 N each,
    the potential's 12 Gaussian terms per pixel and atom in reach."""
    nx, ny, kind = case["nx"], case["ny"], case["kind"]
    N = nx * ny
    S = math.ceil((case["depth"] + 4.0) / case["dz"])
    fft = 5.0 * N * math.log2(N)
    step = 2 * fft + 30.0 * N
    natoms = len(_atoms(case, np.random.default_rng(0))[0])
    ps = case["sx"] / case["nx"]
    # an atom reaches sqrt(5) A: pairs with pixels over the slices it touches
    build = 30.0 * natoms * (math.pi * 3.3 / ps ** 2) * (4.5 + case["dz"]) / case["dz"]
    k = case.get("images", 1)
    if kind in ("steps", "run"):
        return {"bytes": 4.0 * N * S + 8.0 * N, "flops": S * step}
    if kind == "structure":
        return {"bytes": 16.0 * natoms + (4.0 if case["image"] else 8.0) * N, "flops": S * step + build}
    if kind == "raster":
        # every probe's wave is read and written at least once per slice unless it stays on the chip
        return {"bytes": 4.0 * N * S, "flops": case["probes"] * S * step}
    if kind == "phonon":
        return {"bytes": 16.0 * natoms + 8.0 * N, "flops": case["configs"] * (S * step + build)}
    if kind == "forward":
        return {"bytes": 16.0 * natoms + 8.0 * N * k, "flops": S * step + build + k * 2 * fft}
    if kind == "grad":
        return {"bytes": 16.0 * natoms + 4.0 * N * k + (4.0 * N * S if case["want_v"] else 0.0),
                "flops": 2 * S * step + 2 * build + k * 4 * fft}
    if kind == "fd":
        return {"bytes": 4.0 * N * case["steps"] + 8.0 * N, "flops": case["steps"] * step}
    return {"bytes": 8.0 * N + 4.0 * N * k, "flops": (1 + k) * fft}


# ---------------------------------------------------------------------------
# the same in FP64
# ---------------------------------------------------------------------------
class _Setup:
    """Box, frequencies and beam constants, FP32 where they define the problem."""

    def __init__(self, case, atoms):
        self.case, (self.Z, x, y, z), m = case, atoms, _micro(case)
        self.dev = "cuda"
        self.nx, self.ny = case["nx"], case["ny"]
        self.ps, self.dz, V = F(m["ps"]), F(case["dz"]), F(m["kV"])
        self.m = m
        self.off = F(0.0) if case["kind"] == "raster" else F(2.0)
        self.hi = [F(a.max() + F(2)) for a in (x, y, z)]
        self.lo = [F(a.min() - F(2)) for a in (x, y, z)]
        self.top = F(self.hi[2] - self.lo[2])
        self.nz = max(1, int(math.ceil(self.top)))
        self.place(x, y, z)
        pi, e, mm, c2 = F(3.1415926), F(1.6e-19), F(9.11e-31), F(9e16)
        ev = F(F(e * V) * F(1000))
        rest2, rest = F(F(F(2) * mm) * c2), F(mm * c2)
        self.lam = F(F(F(F(6.63e-34) * F(3e8)) / np.sqrt(F(ev * F(rest2 + ev)))) * F(1e10))
        self.sigma = F(F(F(F(2) * pi) / F(F(self.lam * V) * F(1000))) * F(F(rest + ev) / F(rest2 + ev)))
        self.kx, self.ky = self._freq(self.nx), self._freq(self.ny)
        q = [F(float(F(F(k[n // 2 - 1]) / F(2))) ** 2) for k, n in ((self.kx, self.nx), (self.ky, self.ny))]
        self.kmax = np.sqrt(min(q))
        kx, ky = torch.from_numpy(self.kx).to(self.dev), torch.from_numpy(self.ky).to(self.dev)
        self.k2f = (kx * kx)[None, :] + (ky * ky)[:, None]
        self.kxd, self.kyd = kx.double()[None, :], ky.double()[:, None]
        self.k2 = self.kxd ** 2 + self.kyd ** 2
        self.slices = int(math.ceil(F(self.top / self.dz)))
        fp = np.loadtxt(DATA).reshape(-1)[: 103 * 12].reshape(103, 12)
        self.fp = torch.from_numpy(fp).to(self.dev)

    def _freq(self, n):
        size = F(self.ps * F(n))
        i = np.arange(n)
        return np.where(i > n // 2, (i - n).astype(F) / size, i.astype(F) / size).astype(F)

    def place(self, x, y, z):
        self.pos = [F(a - l) for a, l in zip((x, y, z), self.lo)]
        self.bin = np.clip(np.floor(F(self.hi[2] - z)).astype(np.int64), 0, self.nz - 1)

    def propagator(self, dz):
        ph = 3.14159265 * float(dz) * float(self.lam) * self.k2
        return torch.where(torch.sqrt(self.k2f) < float(self.kmax), torch.polar(torch.ones_like(ph), -ph), torch.zeros((), dtype=torch.complex128, device=self.dev))

    def band(self):
        return torch.sqrt(self.k2f) <= float(self.kmax)

    def planes(self, it):
        z = F(self.top - F(self.dz * F(it)))
        sub = [(F(z - F(F(F(k) * self.dz) / F(20))), float(z) - k * float(self.dz) / 20.0) for k in range(1, 21)]
        return z, sub, float(F(self.dz / F(20)))

    def potential(self, z, sub, w, off, grad=None):
        """The slice potential, or with `grad` (dL/dV) the atoms' dL/dx, dL/dy."""
        dev, nx, ny, ps = self.dev, self.nx, self.ny, float(self.ps)
        K = int(math.floor(F(self.top - z)))
        sel = np.nonzero((self.bin >= max(K - 3, 0)) & (self.bin <= min(K + 3, self.nz - 1)))[0]
        V = torch.zeros(ny * nx, dtype=torch.float64, device=dev)
        gx = torch.zeros((len(self.Z), 2), dtype=torch.float64, device=dev)
        width = int(math.ceil(4.4722 / ps)) + 3
        step = max(1, int(6e6) // (width * width))
        o, psf = torch.tensor(off, device=dev), torch.tensor(self.ps, device=dev)
        for s in range(0, len(sel), step):
            ids = sel[s:s + step]
            ax, ay, az = (torch.from_numpy(p[ids]).to(dev) for p in self.pos)
            f = self.fp[torch.from_numpy(self.Z[ids].astype(np.int64) - 1).to(dev)]
            idx = torch.from_numpy(ids).to(dev)
            ix = torch.floor((ax.double() - 2.2361 - float(off)) / ps).long()[:, None] + torch.arange(width, device=dev)
            iy = torch.floor((ay.double() - 2.2361 - float(off)) / ps).long()[:, None] + torch.arange(width, device=dev)
            dxf = (o + ix.float() * psf) - ax[:, None]
            dyf = (o + iy.float() * psf) - ay[:, None]
            rho_f = (dxf * dxf)[:, None, :] + (dyf * dyf)[:, :, None]
            dx = float(off) + ix.double() * ps - ax.double()[:, None]
            dy = float(off) + iy.double() * ps - ay.double()[:, None]
            inside = ((ix >= 0) & (ix < nx))[:, None, :] & ((iy >= 0) & (iy < ny))[:, :, None]
            inside &= rho_f < 5.0
            at, py, pxi = torch.nonzero(inside, as_tuple=True)
            rf, rho = rho_f[at, py, pxi], dx[at, pxi] ** 2 + dy[at, py] ** 2
            pix = iy[at, py] * nx + ix[at, pxi]
            acc = torch.zeros_like(rho)
            for zf, zd in sub:
                dzf = torch.tensor(zf, device=dev) - az
                near = torch.nonzero(rf + (dzf * dzf)[at] < 5.0, as_tuple=True)[0]
                if not len(near):
                    continue
                a = at[near]
                r2 = rho[near] + ((zd - az.double()) ** 2)[a]
                r = torch.sqrt(r2).clamp(min=0.25)
                t = torch.zeros_like(r)
                for k in range(3):
                    A, B, C, D = f[a, 2 * k], f[a, 2 * k + 1], f[a, 6 + 2 * k], f[a, 7 + 2 * k]
                    b = 2.0 * 3.141592654 * torch.sqrt(B)
                    L = 150.4121417 * A * torch.exp(-b * r)
                    q = 3.141592654 ** 2 / D
                    G = 266.5157269 * C * D ** -1.5 * torch.exp(-q * r * r)
                    t += L / r + G if grad is None else -L * (b * r + 1.0) / (2.0 * r ** 3) - q * G
                if grad is not None:
                    t = torch.where(r2 < 0.0625, torch.zeros_like(t), t)
                acc[near] += w * t
            if grad is None:
                V.index_add_(0, pix, acc)
            else:
                t = -2.0 * acc * grad.reshape(-1)[pix]
                gx.index_add_(0, idx[at], torch.stack([t * dx[at, pxi], t * dy[at, py]], 1))
        return V.reshape(ny, nx) if grad is None else gx

    def stack(self, slices):
        for it in range(1, slices + 1):
            z, sub, w = self.planes(it)
            yield self.potential(z, sub, w, self.off)

    def ctf(self, df):
        m, lam, Cs = self.m, float(self.lam), float(F(self.m["Cs"]))
        beta, delta = float(F(F(m["beta"]) / F(1000))), float(F(m["delta"]))
        q = F(F(F(m["ap"]) * F(0.001)) / self.lam)
        k = torch.sqrt(self.k2)
        a1 = 3.141593 * k * lam * 2.0 * df + 2.0 * 3.141593 * lam ** 3 * Cs * self.k2 * k
        es = torch.exp(-beta ** 2 / (4.0 * lam ** 2) * a1 ** 2)
        ed = torch.exp(-0.25 * delta ** 2 * 3.141593 ** 2 * self.k2 ** 2 * lam ** 2)
        chi = 3.1415926 * lam * self.k2 * (0.5 * Cs * lam ** 2 * self.k2 + df)
        return torch.where(self.k2f < float(F(q * q)), torch.polar(es * ed, -chi), torch.zeros((), dtype=torch.complex128, device=self.dev))

    def image(self, spectrum, df):
        return torch.fft.ifft2(self.ctf(df) * spectrum).abs() ** 2


def _wave(s, slices, stack=None):
    P = s.propagator(s.dz)
    psi = torch.ones((s.ny, s.nx), dtype=torch.complex128, device=s.dev)
    for V in (s.stack(slices) if stack is None else stack):
        psi = torch.fft.ifft2(P * torch.fft.fft2(psi * torch.exp(1j * float(s.sigma) * V)))
    return psi


def _philox_normals(seed, config, n):
    """Displacement normals per atom: Philox4x32-10, counter (atom, pass, 0x5EED, 0)."""
    c = [np.arange(n, dtype=np.uint64), np.full(n, config, np.uint64), np.full(n, 0x5EED, np.uint64), np.zeros(n, np.uint64)]
    k, low = [seed & 0xFFFFFFFF, seed >> 32], np.uint64(0xFFFFFFFF)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k[0]), p1 & low, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k[1]), p0 & low]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    u = [(v.astype(np.float64) + 0.5) * 2.0 ** -32 for v in c]
    m0, m1 = np.sqrt(-2.0 * np.log(u[0])), np.sqrt(-2.0 * np.log(u[2]))
    t0, t1 = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    return m0 * np.cos(t0), m0 * np.sin(t0), m1 * np.cos(t1)


def exact(case, seed):
    kind = case["kind"]
    # pixel, atom and plane triples of the potential (20 planes a slice)
    S = math.ceil((case["depth"] + 4.0) / case["dz"])
    natoms = len(_atoms(case, np.random.default_rng(0))[0])
    triples = natoms * math.pi * 3.3 / (case["sx"] / case["nx"]) ** 2 * 4.5 / case["dz"] * 20
    if triples * case.get("configs", 1) * (2 if kind == "grad" else 1) > 6e10:
        return None
    d = _inputs(case, seed)
    s = _Setup(case, d["atoms"])
    if kind in ("steps", "run", "structure"):
        psi = _wave(s, s.slices)
        if not case.get("image"):
            return {"wave": psi}
        return {"image": s.image(torch.fft.fft2(psi), float(F(s.m["df"])))}
    if kind == "images":
        spec = torch.fft.fft2(_wave(s, s.slices))
        return {"images": torch.stack([s.image(spec, float(df)) for df in d["defoci"]])}
    if kind == "raster":
        P, lam = s.propagator(s.dz), float(s.lam)
        kf = torch.sqrt(s.k2f)
        apert = float(F(float(F(s.m["ap"])) * 0.001 / lam))
        trans = [torch.exp(1j * float(s.sigma) * V) for V in s.stack(s.slices)]
        ki, ko = (F(F(F(v) * F(0.001)) / s.lam) for v in (70.0, 200.0))
        ring = (s.k2f >= float(F(ki * ki))) & (s.k2f < float(F(ko * ko)))
        out = []
        for px, py in zip(d["px"].tolist(), d["py"].tolist()):
            ph = 2.0 * 3.14159265 * float(s.ps) * (s.kxd * px + s.kyd * py)
            psi = torch.fft.ifft2(torch.where(kf < apert, torch.polar(torch.ones_like(ph), ph), torch.zeros((), dtype=torch.complex128, device=s.dev)))
            psi = psi / psi.abs().sum()
            for t in trans:
                psi = torch.fft.ifft2(P * torch.fft.fft2(psi * t))
            out.append((torch.fft.fft2(psi).abs() ** 2)[ring].sum() / (s.nx * s.ny))
        return {"signal": torch.stack(out)}
    if kind == "phonon":
        diff = torch.zeros((s.ny, s.nx), dtype=torch.float64, device=s.dev)
        image = torch.zeros_like(diff)
        for k in range(case["configs"]):
            moved = [F(a.astype(np.float64) + float(F(0.076)) * q) for a, q in zip(d["atoms"][1:], _philox_normals(seed + 1, k, len(s.Z)))]
            s.place(*moved)
            spec = torch.fft.fft2(_wave(s, s.slices))
            diff += torch.roll(spec.abs(), (s.ny // 2, s.nx // 2), (0, 1))
            image += s.image(spec, float(F(s.m["df"]))) / case["configs"]
        return {"diffraction": diff, "image": image}
    if kind in ("grad", "forward"):
        V = torch.stack(list(s.stack(s.slices))).requires_grad_(kind == "grad")
        spec = torch.fft.fft2(_wave(s, s.slices, V))
        images = [s.image(spec, float(df)) for df in d["defoci"]]
        T = torch.from_numpy(d["targets"]).to(s.dev).double()
        loss = sum(((im - t) ** 2).sum() for im, t in zip(images, T))
        if kind == "forward":
            return {"loss": float(loss), "images": torch.stack(images)}
        loss.backward()
        gxy = torch.zeros((len(s.Z), 2), dtype=torch.float64, device=s.dev)
        for it in range(1, s.slices + 1):
            z, sub, w = s.planes(it)
            gxy += s.potential(z, sub, w, s.off, V.grad[it - 1])
        out = {"loss": float(loss), "dxy": gxy}
        if case["want_v"]:
            out["dv"] = V.grad
        return out
    if kind == "fd":
        dz, lam, sig = F(case["fd_dz"]), float(s.lam), float(s.sigma)
        a = 2.0 * 3.14159 * float(dz) / lam
        rc, ratio = 1.0 / (1.0 + 1j * a), (1.0 - 1j * a) / (1.0 + 1j * a)
        kv = float(dz) ** 2 * 4.0 * 3.14159 * sig / lam
        lap = -4.0 * 3.14159 ** 2 * s.k2 * float(dz) ** 2
        band = s.band().double()
        before = torch.ones((s.ny, s.nx), dtype=torch.complex128, device=s.dev)
        psi = before.clone()
        for it in range(1, case["steps"] + 1):
            z = F(s.top - F(dz * F(it)))
            V = s.potential(z, [(z, float(z))], 1.0, F(0.0))
            V = torch.fft.ifft2(band * torch.fft.fft2(V)).real
            grad = torch.fft.ifft2(lap * torch.fft.fft2(psi))
            nxt = rc * (2.0 * psi - grad - kv * V * psi) - ratio * before
            before, psi = psi, torch.fft.ifft2(band * torch.fft.fft2(nxt))
        return {"wave": psi}
    return None
