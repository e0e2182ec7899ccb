"""The work whose speed is measured, through the Python mirror of the C-ABI (`g3d.Simulation`).

A user of this library marches a window: load a bunch, make the start field, then s-step after s-step, reading the
diagnostics sums (a line of diag.txt) as the run goes. The cases are such s-steps over the range of sizes and options
that the configurations, tests and benchmark of this repository use:

  wake      frozen-bunch wake in vacuum (the benchmark's workload 1): beam push, deposit, transforms, march, real fields
  wave      a dense bunch in an oblique analytic plane wave (workload 2): the same with the sponge and RK4 sub-steps
  exchange  a step coupled to a host program: the particle records go in, step, and come back (the benchmark's e2e)
  lwfa      laser wakefield with streaming plasma (workload 3, the example deck): the half-cell march with its passes
  gas       ionization injection on free-hand y and zeta grids (workload 5): neutral gas, ADK ionization, walls
  adjoint   an objective and its gradients (workload 4): start field, K s-steps, the reverse sweep; with plasma or not

in the FP64 and the mixed form. Outputs are the library's own device arrays (spectra in their half layout, real fields),
the diagnostics sums, and the particles or gradients where the call returns them. `exact` restates the step in 64 bits
with torch.
"""
import importlib
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "gem-pic-3d_b200"))
g3d = importlib.import_module("g3d")
configs = importlib.import_module("g3d.configs")

SIZES = (16, 24, 32, 48, 64, 96, 128, 192, 256)


def listed():
    return [
        # the smallest call: a test-size wake, launches and host latency count
        dict(name="wake 32x32x64", kind="wake", nx=32, ny=32, nz=64, n=8192, form="fp64"),
        # workload 1 in full: the CPU-runnable deck, an ordinary vacuum step
        dict(name="wake 64x64x256", kind="wake", nx=64, ny=64, nz=256, n=262144, form="fp64"),
        # workload 2 in full, both forms: the large vacuum step
        dict(name="wave 128x128x1024", kind="wave", nx=128, ny=128, nz=1024, n=1048576, form="fp64"),
        dict(name="wave 128x128x1024 mixed", kind="wave", nx=128, ny=128, nz=1024, n=1048576, form="mixed"),
        # ragged sizes (three times a power of two, odd slice and particle counts) coupled to a host program
        dict(name="exchange 96x48x301", kind="exchange", nx=96, ny=48, nz=301, n=100003, form="fp64"),
        # a small plasma run (test size): a chain of short launches; electrons only, smoothed current
        dict(name="lwfa 32x32x160 mixed", kind="lwfa", nx=32, ny=32, nz=160, n=5000, form="mixed", ppc=2, ions=False,
             passes=2, smooth=0.4),
        # the size of the example LWFA deck (64 x 64 modes, 1201 slices, 2 x 2 electrons a cell, two passes)
        dict(name="lwfa 64x64x1201", kind="lwfa", nx=64, ny=64, nz=1201, n=100000, form="fp64", ppc=2, ions=True,
             passes=2, smooth=0.0),
        # workload 3 on a shorter window in the FP64 form
        dict(name="lwfa 256x256x384", kind="lwfa", nx=256, ny=256, nz=384, n=1048576, form="fp64", ppc=2, ions=True,
             passes=2, smooth=0.0),
        # workload 3 in full, the headline: mixed form
        dict(name="lwfa 256x256x2048 mixed", kind="lwfa", nx=256, ny=256, nz=2048, n=4194304, form="mixed", ppc=2,
             ions=True, passes=2, smooth=0.0),
        # workload 5's grids on a short window with a thinner lattice: ionization, walls, graded zeta
        dict(name="gas 256x192x256 mixed", kind="gas", nx=256, half=96, nz=256, form="mixed", ppc=3),
        # workload 4 without its plasma: forward and backward, fewer steps
        dict(name="adjoint 64x64x512", kind="adjoint", nx=64, ny=64, nz=512, n=65536, form="fp64", steps=10,
             plasma=False),
        # workload 4 with its plasma, mixed form, a shorter window and two steps
        dict(name="adjoint plasma 64x64x256 mixed", kind="adjoint", nx=64, ny=64, nz=256, n=65536, form="mixed", steps=2,
             plasma=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("wake", "wave", "exchange", "lwfa", "lwfa", "gas", "adjoint"))
    form = rng.choice(("fp64", "mixed"))
    if kind == "gas":
        return dict(kind=kind, nx=rng.choice((64, 96, 128, 256)), half=rng.choice((72, 80, 96)), nz=_log_int(rng, 140, 260),
                    form=form, ppc=rng.randint(1, 3))
    if kind == "adjoint":
        nx, ny = rng.choice((16, 32, 48, 64)), rng.choice((16, 32, 48, 64))
        return dict(kind=kind, nx=nx, ny=ny, nz=_log_int(rng, 192, 512), n=_log_int(rng, 2000, 65536), form=form,
                    steps=rng.randint(1, 3), plasma=rng.random() < 0.5)
    nx = rng.choice(SIZES)
    ny = rng.choice([s for s in SIZES if nx <= 4 * s and s <= 4 * nx])
    if kind == "lwfa":
        # no more than a quarter of the headline's half-cells at its transverse size
        nz = _log_int(rng, 96, 700)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, n=_log_int(rng, 2000, 1000000), form=form, ppc=rng.randint(1, 2),
                    ions=rng.random() < 0.6, passes=rng.choice((1, 2, 2, 3)), smooth=rng.choice((0.0, 0.4)))
    n = _log_int(rng, 3000, 300000 if kind == "exchange" else 1500000)
    return dict(kind=kind, nx=nx, ny=ny, nz=_log_int(rng, 48, 1100 if nx * ny <= 16384 else 400), n=n, form=form)


# ---------------------------------------------------------------- configurations
def config(case, rng):
    """The run of a case: the repository's configuration of its kind at the case's sizes, laser phase from rng."""
    k = case["kind"]
    if k == "gas":
        c = configs.config5(nx=case["nx"], half=case["half"], nzeta=case["nz"], ppc=case["ppc"], steps=100)
        c.plasma["seed"] = int(rng.integers(1, 1 << 30))
    elif k == "adjoint":
        c = configs.config4(nx=case["nx"], ny=case["ny"], nzeta=case["nz"], nmacro=case["n"], steps=case["steps"],
                            plasma=case["plasma"])
    elif k == "lwfa":
        # the workload's own step; a window of 51 at least, which holds the laser and the witness
        c = configs.config3(nx=case["nx"], ny=case["ny"], nzeta=case["nz"], nmacro=case["n"],
                            h=max(0.2, 51.0 / (case["nz"] - 1)))
        c.plasma.update(ppc_x=case["ppc"], ppc_y=case["ppc"], iterations=case["passes"], smooth_length=case["smooth"])
        c.ions = c.ions if case["ions"] else []
    elif k == "wake":
        c = configs.config1(nx=case["nx"], ny=case["ny"], nzeta=case["nz"], nmacro=case["n"])
    else:
        c = configs.config2(nx=case["nx"], ny=case["ny"], nzeta=case["nz"], nmacro=case["n"])
    phase = float(rng.uniform(0, 2 * math.pi))
    for g in c.glasers:
        g.update(cep=phase, pol_angle=0.4)
    if c.params.get("laser_on"):
        c.params["cep"] = phase
    return c


def records(cfg, rng):
    """The bunch of a configuration as particle records (the Gaussian bunch that g3d_load_bunches samples, drawn by
    numpy), those outside the window moved to its ends."""
    b = dict(configs.default_bunch(), **cfg.bunches[0])
    n = b["nmacro"]
    Lu, nc = configs.units(cfg.params["lambda0"])
    p = np.zeros(n, dtype=g3d.PARTICLE_DTYPE)
    z = b["sigz"] * rng.standard_normal(n)
    p["px"] = b["emitx"] / b["sigx"] * rng.standard_normal(n)
    p["py"] = b["emity"] / b["sigy"] * rng.standard_normal(n)
    p["pz"] = math.sqrt(b["gamma"] ** 2 - 1) * (1 + b["espread"] * rng.standard_normal(n))
    vz = p["pz"] / np.sqrt(1 + p["px"] ** 2 + p["py"] ** 2 + p["pz"] ** 2)
    p["x"] = b["x0"] + b["sigx"] * rng.standard_normal(n) - p["px"] / p["pz"] * z + 0.5 * cfg.Lx
    p["y"] = b["y0"] + b["sigy"] * rng.standard_normal(n) - p["py"] / p["pz"] * z + 0.5 * cfg.Ly
    p["zeta"] = b["zeta_center"] + z / vz
    p["w"] = b["charge_C"] / configs.E_SI / n / (nc * Lu ** 3)
    p["q"] = p["qm"] = b["q"]
    p["alive"] = 1
    p["id"] = np.arange(n)
    p["zeta"] = np.clip(p["zeta"], 0.0, cfg.zeta[-1] - 1e-3 * cfg.h)
    return p


def inputs(case, seed):
    rng = np.random.default_rng(seed)
    cfg = config(case, rng)
    return cfg, (records(cfg, rng) if cfg.bunches else None)


# ---------------------------------------------------------------- a pass
class _View:
    """A device array of a simulation as torch sees it; keeps the simulation alive."""

    def __init__(self, sim, ptr, shape, typestr):
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _array(state, name):
    """The library's storage of an array: spectra [plane][j][kx <= nx/2] as pairs, F [comp][fl][j][ix]."""
    sim = state["sim"]
    ptr = sim.device_ptr(name)
    if ptr not in state["views"]:
        N, nx, ny = sim.N, sim.nx, sim.ny
        if name == "F":
            shape, typ = (6, N + 2, ny, nx), "<f4"
        elif name.startswith("rho"):
            shape, typ = (N, nx + ny), "<f8"
        else:
            narrow = sim.precision == "mixed" and sim.cfg.ynode is None and not name.startswith("R")
            shape, typ = (N + (1 if name.startswith("j") else 0), ny, nx // 2 + 1, 2), "<f4" if narrow else "<f8"
        state["views"][ptr] = torch.as_tensor(_View(sim, ptr, shape, typ), device="cuda")
    return state["views"][ptr]


def prepare(case, seed):
    cfg, parts = inputs(case, seed)
    sim = g3d.Simulation(cfg, precision=case["form"])
    state = {"kind": case["kind"], "sim": sim, "parts": parts, "views": {}}
    if case["kind"] == "adjoint":
        if case["form"] == "fp64":
            sim.set_exact_fields(True)
        sim.set_laser_modes(np.ones((cfg.ny, cfg.nx // 2 + 1)))
        state["steps"] = case["steps"]
        return state
    if parts is not None:
        sim.set_particles(parts)
    sim.init_fields()
    return state


def run(state):
    sim = state["sim"]
    if state["kind"] == "adjoint":
        sim.set_particles(state["parts"])
        sim.init_fields()
        J, gm, gp = sim.adjoint(state["steps"])
        return {"J": J, "modes": gm, "momenta": gp}
    if state["kind"] == "exchange":
        sim.set_particles(state["parts"])
        sim.step()
        state["parts"] = q = sim.host_particles()
        return {"sums": sim.diagnostics_sums(), "F": _array(state, "F"),
                **{f: q[f] for f in ("x", "y", "zeta", "px", "py", "pz")}}
    sim.step()
    names = ["Rx", "Ry", "j0x", "j0y", "F"]
    names += ["rho_lines"] if sim.cfg.plasma is not None else ["jkz"]
    return {"sums": sim.diagnostics_sums(), **{a: _array(state, a) for a in names}}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    nx, nz = case["nx"], case["nz"]
    ny = 2 * case["half"] if case["kind"] == "gas" else case["ny"]
    G, Gh = nx * ny * nz, ny * (nx // 2 + 1) * nz
    n = case.get("n", 0)
    cz = 16 if case["form"] == "fp64" or case["kind"] in ("gas", "adjoint") else 8
    # a step: F read and written; R read and written; E_z, B_z, j0 read; E_z, B_z, L, j0, j_z written; the beam's
    # six coordinates read and written, its weight, charge and state read
    step = 2 * 24 * G + (4 * 16 + 4 * cz + 7 * cz) * Gh + (2 * 48 + 28) * n
    # five transforms forward and six back (the sponge two more each way), the march's ~150 operations per mode, RK4
    # and the deposit ~2500 per beam particle
    fft = 5 * G * math.log2(nx * ny) * 5.5
    flops = fft + 150 * Gh + 2500 * n
    if case["kind"] == "gas" or case.get("plasma") or case["kind"] == "lwfa":
        # the streaming plasma's state, read once and written once per half-cell, and its current of level s0
        ppc = case.get("ppc", 2)
        per = 2 if case["kind"] == "gas" or case.get("ions") else 1
        S = nx * ny * ppc * ppc * per
        passes = case.get("passes", 2)
        step += nz * S * (11 * 8 + 7 * 8) + 2 * 3 * 16 * Gh
        flops += passes * (nz * S * 500.0 + fft)
    if case["kind"] == "adjoint":
        k = case["steps"]
        # each step forward, each step's fields and beam read again and their adjoints carried back
        return {"bytes": float(3 * k * step), "flops": float(3 * k * flops)}
    if case["kind"] == "exchange":
        step += 2 * 104 * n
    return {"bytes": float(step), "flops": float(flops)}


def tolerance(case):
    # About four times the distance from `exact` on the listed cases (vacuum FP64 6e-8 by the float F that the push
    # gathers, mixed 2e-7; plasma FP64 3.5e-5, mixed 1e-3 in the densities at the axis, which the trapped electrons
    # amplify); gas and adjoint: about four times the distance between the two forms (1.3e-6 and 4e-9), with room for
    # an ionization event that falls the other way and for shorter, coarser windows.
    if case["kind"] == "adjoint":
        return {"rel": 1e-7, "max": 1e-6}
    if case["kind"] == "gas":
        return {"rel": 5e-6, "max": 1e-3}
    if case["kind"] == "lwfa":
        return {"rel": 1.5e-4, "max": 2e-2} if case["form"] == "fp64" else {"rel": 4e-3, "max": 1e-1}
    return {"rel": 2.5e-7, "max": 1.5e-5} if case["form"] == "fp64" else {"rel": 2e-6, "max": 1e-4}


# ---------------------------------------------------------------- the same in 64 bits
class _March:
    """One window of the march on a Fourier y grid with uniform zeta, in torch's 64-bit arithmetic: the start field
    and one s-step, in vacuum or with streaming electrons and mobile ions."""

    def __init__(self, cfg, parts):
        self.c, self.p = cfg, dict(configs.default_params(), **cfg.params)
        self.dev = "cuda"
        nx, ny, N = cfg.nx, cfg.ny, cfg.nzeta
        self.nx, self.ny, self.N, self.H = nx, ny, N, nx // 2 + 1
        self.dx, self.dy = cfg.Lx / nx, cfg.Ly / ny
        self.X0, self.Y0 = -0.5 * cfg.Lx, -0.5 * cfg.Ly
        self.h = float(cfg.zeta[-1]) / (N - 1)
        T = lambda v: torch.tensor(v, dtype=torch.float64, device=self.dev)  # noqa: E731
        kx = 2 * math.pi * np.arange(self.H) / cfg.Lx
        my = np.arange(ny)
        my = np.where(my <= ny // 2, my, my - ny)
        ky = 2 * math.pi * my / cfg.Ly
        fx, fy = np.cos(0.5 * kx * self.dx) ** 2, np.cos(0.5 * ky * self.dy) ** 2
        fx[2 * np.arange(self.H) == nx], fy[2 * np.arange(ny) == ny] = 0, 0
        self.filt = T(fy[:, None] * fx[None, :])
        self.k2s = T(ky[:, None] ** 2 + kx[None, :] ** 2)
        kxd, kyd = np.where(2 * np.arange(self.H) == nx, 0, kx), np.where(2 * np.arange(ny) == ny, 0, ky)
        self.ix = 1j * T(np.broadcast_to(kxd[None, :], (ny, self.H)).copy())
        self.iy = 1j * T(np.broadcast_to(kyd[:, None], (ny, self.H)).copy())
        self.k2 = T(kyd[:, None] ** 2 + kxd[None, :] ** 2)

        def mask(n, d, L, w):
            e = np.minimum(np.arange(n) * d, L - np.arange(n) * d)
            return np.where(e < w, 1 - self.p["sponge_rate"] * (1 - e / w) ** 2, 1.0) if w > 0 else np.ones(n)
        self.mask = T(mask(ny, self.dy, cfg.Ly, self.p["sponge_y"])[:, None] * mask(nx, self.dx, cfg.Lx, self.p["sponge"])[None, :])
        z = lambda n: torch.zeros(n, ny, self.H, dtype=torch.complex128, device=self.dev)  # noqa: E731
        self.R = [z(N), z(N)]
        self.E, self.B = z(N), z(N)
        self.L = [z(N), z(N)]
        self.j0 = [z(N + 1), z(N + 1)]
        self.jk = None
        self.F = torch.zeros(6, N + 2, ny, nx, dtype=torch.float64, device=self.dev)
        self.lines = None
        self.q = [T(np.ascontiguousarray(parts[f])) for f in ("x", "y", "zeta", "px", "py", "pz")]
        self.w, self.qm = T(np.ascontiguousarray(parts["w"])), T(np.ascontiguousarray(parts["qm"]))
        self.alive = torch.ones_like(self.w, dtype=torch.bool)
        self.trapped = (0, 0.0)

    @staticmethod
    def tsc(x, d, n):
        xi = x / d
        i0 = torch.floor(xi + 0.5)
        f = xi - i0
        w = torch.stack([0.5 * (0.5 - f) ** 2, 0.75 - f * f, 0.5 * (0.5 + f) ** 2])
        i = torch.stack([i0 - 1, i0, i0 + 1]).to(torch.int64) % n
        return i, w

    def stencil(self, x, y):
        """[9, n] points and weights of the transverse TSC."""
        ix, wx = self.tsc(x, self.dx, self.nx)
        iy, wy = self.tsc(y, self.dy, self.ny)
        return ((iy[:, None] * self.nx + ix[None, :]).reshape(9, -1), (wy[:, None] * wx[None, :]).reshape(9, -1))

    # ------------------------------------------------------------ currents
    def currents(self, keep0):
        N, ny, nx = self.N, self.ny, self.nx
        x, y, zeta, px, py, pz = self.q
        m = torch.floor(zeta / self.h).to(torch.int64)
        ok = self.alive & (m >= 0) & (m <= N - 2)
        k, w9 = self.stencil(x[ok], y[ok])
        f = self.w[ok] * self.qm[ok] / (self.h * self.dx * self.dy)
        J = []
        for v in (px / pz, py / pz, torch.ones_like(px)):
            a = torch.zeros((N + 3) * ny * nx, dtype=torch.float64, device=self.dev)
            for s in range(9):
                a.index_add_(0, (m[ok] + 2) * (ny * nx) + k[s], f * w9[s] * v[ok])
            J.append(a.view(N + 3, ny, nx))
        filt = self.filt.clone()
        if not keep0:
            filt[0, 0] = 0
        out = []
        for a in J:
            o = torch.zeros(N + 1, ny, self.H, dtype=torch.complex128, device=self.dev)
            for c in range(1, N, 64):                       # half-cells 0 .. N-2 at planes 1 .. N-1
                e = min(N, c + 64)
                v = 0.25 * a[c:e] + 0.5 * a[c + 1:e + 1] + 0.25 * a[c + 2:e + 2]
                o[c:e] = filt * torch.fft.rfft2(v)
            out.append(o)
        self.jk = out

    # ------------------------------------------------------------ the march
    def march_slice(self, n, D, R, E, B):
        """Slice n from its level-s0 values R, E, B; the slice above is final."""
        a, b, jk, j0 = self.ix, self.iy, self.jk, self.j0
        J = [0.5 * (j0[c][n] + jk[c][n] + j0[c][n + 1] + jk[c][n + 1]) for c in (0, 1)]
        Rx = R[0] + D * (a * E + b * B) - D * J[0]
        Ry = R[1] + D * (b * E - a * B) - D * J[1]
        if n == self.N - 1:
            self.R[0][n], self.R[1][n] = Rx, Ry
            for t in (self.E, self.B, *self.L):
                t[n] = 0
            return
        pRx, pRy, pE, pB, pLx, pLy = (t[n + 1] for t in (*self.R, self.E, self.B, *self.L))
        h, q = self.h, 0.25 * self.h
        Lx = pLx - q * (a * pE - b * pB) - 0.5 * h * jk[0][n + 1]
        Ly = pLy - q * (a * pB + b * pE) - 0.5 * h * jk[1][n + 1]
        C = 0.5 * (a * (pRy + pLy) - b * (pRx + pLx))
        Q = 0.5 * (b * (pLy - pRy) - a * (pRx - pLx))
        den = 1 + q * (D + q) * self.k2
        Bn = (pB - 0.5 * h * C - q * (a * (Ry + Ly) - b * (Rx + Lx))) / den
        En = (pE - 0.5 * h * Q - q * (a * (Lx - Rx) + b * (Ly - Ry)) - h * jk[2][n + 1]) / den
        self.E[n], self.B[n] = En, Bn
        self.R[0][n] = Rx + D * (a * En + b * Bn)
        self.R[1][n] = Ry + D * (b * En - a * Bn)
        self.L[0][n] = Lx - q * (a * En - b * Bn)
        self.L[1][n] = Ly - q * (a * Bn + b * En)

    def march(self, D):
        for n in range(self.N - 1, -1, -1):
            self.march_slice(n, D, [self.R[0][n], self.R[1][n]], self.E[n], self.B[n])

    def real(self, c, e):
        """Real fields of the slices c .. e - 1."""
        s = (self.ny, self.nx)
        r1, r2, l1, l2 = (torch.fft.irfft2(t[c:e], s=s) for t in (*self.R, *self.L))
        self.F[0, c:e], self.F[1, c:e] = 0.5 * (r1 + l1), 0.5 * (r2 + l2)
        self.F[3, c:e], self.F[4, c:e] = 0.5 * (l2 - r2), 0.5 * (r1 - l1)
        self.F[2, c:e], self.F[5, c:e] = torch.fft.irfft2(self.E[c:e], s=s), torch.fft.irfft2(self.B[c:e], s=s)

    def sponge_and_real(self):
        N, h, jz = self.N, self.h, self.jk[2]
        if self.p["sponge"] > 0 or self.p["sponge_y"] > 0:
            zero = torch.zeros_like(jz[:1])
            rho = torch.cat([zero, 0.5 * (jz[:N] + jz[1:N + 1]), zero])
            ik2 = torch.where(self.k2 > 0, 1 / self.k2.clamp_min(1e-300), torch.zeros_like(self.k2))
            for c in range(0, N, 64):
                e = min(N, c + 64)
                r = rho[c + 1:e + 1]
                d2 = self.gm2 * (rho[c + 2:e + 2] - 2 * r + rho[c:e]) / (h * h)
                psi = (r + d2 * ik2) * ik2
                for k, g in ((0, self.ix), (1, self.iy)):
                    bound = -(1 + self.beta) * g * psi
                    s = self.mask * torch.fft.irfft2(self.R[k][c:e] - bound, s=(self.ny, self.nx))
                    self.R[k][c:e] = torch.fft.rfft2(s) + bound
        for c in range(0, N, 64):
            self.real(c, min(N, c + 64))

    # ------------------------------------------------------------ the start field
    def comoving(self, beta):
        N, h = self.N, self.h
        gm2 = 1 - beta * beta
        off, dg = -gm2 / (h * h), self.k2 + 2 * gm2 / (h * h)
        live = dg != 0
        c = torch.zeros_like(self.k2)
        d = torch.zeros_like(self.ix)
        cs, ds = [], []
        for n in range(N):
            den = torch.where(live, dg - off * c, torch.ones_like(dg))
            rhs = 0.5 * (self.jk[2][n] + self.jk[2][n + 1]) / beta
            d = torch.where(live, (rhs - off * d) / den, torch.zeros_like(d))
            c = torch.where(live, off / den, torch.zeros_like(c))
            cs.append(c)
            ds.append(d)
        psi = torch.zeros_like(d)
        for n in range(N - 1, -1, -1):
            psi = ds[n] - cs[n] * psi
            self.R[0][n], self.R[1][n] = -(1 + beta) * self.ix * psi, -(1 + beta) * self.iy * psi

    def start(self):
        pz, g = self.q[5], torch.sqrt(1 + self.q[3] ** 2 + self.q[4] ** 2 + self.q[5] ** 2)
        # 1 - beta is a small difference: summed as such
        omv = (1 + self.q[3] ** 2 + self.q[4] ** 2) / (g * (g + pz))
        omb = float((self.w * omv).sum() / self.w.sum())
        self.beta, self.gm2 = 1 - omb, omb * (2 - omb)
        self.currents(False)
        self.comoving(self.beta)
        keep = [r.clone() for r in self.R]
        self.comoving(1.0)
        diff = [a - b for a, b in zip(keep, self.R)]
        for _ in range(3):
            for t in (self.E, self.B, *self.j0):
                t.zero_()
            self.march(100 * self.p["dz"])
        for r, d in zip(self.R, diff):
            r += d
        x = torch.arange(self.nx, device=self.dev) * self.dx + self.X0
        y = torch.arange(self.ny, device=self.dev) * self.dy + self.Y0
        zeta = torch.tensor(self.c.zeta, device=self.dev)
        for L in self.c.glaser_structs():
            qb = complex(1.0, -L.z_focus / (0.5 * L.kL * L.waist ** 2))
            prof = torch.exp(-(x[None, :] ** 2 + y[:, None] ** 2) / (L.waist ** 2 * qb)) / qb
            P, Q = torch.fft.rfft2(prof.real.contiguous()), torch.fft.rfft2(prof.imag.contiguous())
            d = zeta - L.zeta_c
            env = torch.exp(-2 * math.log(2.0) * d * d / L.tau ** 2)
            env = torch.where(env.abs() < 1e-12, torch.zeros_like(env), env)
            cn = L.a0 * L.kL * env * torch.exp(1j * (L.kL * d + L.cep))
            for n in range(self.N):
                u = 2 * (cn[n].real * P - cn[n].imag * Q)
                self.R[0][n] += math.cos(L.pol_angle) * u
                self.R[1][n] += math.sin(L.pol_angle) * u
        self.march(0.0)
        self.sponge_and_real()
        self.j0 = [self.jk[0].clone(), self.jk[1].clone()]

    # ------------------------------------------------------------ the beam push
    def wave(self, x, z, t):
        p = self.p
        sx, cz = math.sin(p["theta"]), math.cos(p["theta"])
        xi = t - sx * x - cz * z - p["eta_c"]
        hf, rp = 0.5 * p["flat_length"], p["ramp_length"]
        u = (hf + rp - xi.abs()) / rp
        sn, cs = torch.sin(0.5 * math.pi * u), torch.cos(0.5 * math.pi * u)
        flat, live = xi.abs() <= hf, xi.abs() < hf + rp
        g = torch.where(flat, torch.ones_like(u), sn * sn)
        gp = torch.where(flat, torch.zeros_like(u), -torch.sign(xi) * (math.pi / rp) * sn * cs)
        ph = p["kL"] * xi + p["cep"]
        d = torch.where(live, p["a0"] * (gp * torch.cos(ph) - p["kL"] * g * torch.sin(ph)), torch.zeros_like(u))
        Ex, Ez = -d * cz, d * sx
        return Ex, Ez, cz * Ex - sx * Ez                     # p polarisation: E_x, E_z, B_y

    def rhs(self, Y, z, qm):
        x, y, zeta, px, py, pz = Y
        g = torch.sqrt(1 + px * px + py * py + pz * pz)
        t = zeta / self.h
        n = torch.floor(t).to(torch.int64)
        f = t - n
        ok = (n >= 0) & (n <= self.N)
        n = n.clamp(0, self.N)
        k, w = self.stencil(torch.remainder(x, self.c.Lx), torch.remainder(y, self.c.Ly))
        nk = self.nx * self.ny
        F = self.F.view(6, -1)
        f = torch.where(ok, f, torch.zeros_like(f))
        e = torch.zeros(6, len(x), dtype=torch.float64, device=self.dev)
        for s in range(9):
            e += w[s] * ((1 - f) * F[:, n * nk + k[s]] + f * F[:, (n + 1) * nk + k[s]])
        e = torch.where(ok, e, torch.zeros_like(e))
        E, B = list(e[:3]), list(e[3:])
        if self.p["laser_on"]:
            ex, ez, by = self.wave(x + self.X0, z, z - (zeta - self.p["zeta_center"]))
            E[0], E[2], B[1] = E[0] + ex, E[2] + ez, B[1] + by
        i = 1 / pz
        return torch.stack([px * i, py * i, -(1 + px * px + py * py) / (g + pz) * i,
                            qm * (g * E[0] + py * B[2] - pz * B[1]) * i, qm * (g * E[1] + pz * B[0] - px * B[2]) * i,
                            qm * (g * E[2] + px * B[1] - py * B[0]) * i])

    def push(self, s0, s1):
        Y, z = torch.stack(self.q), torch.full_like(self.w, s0)
        while True:
            a = torch.nonzero(z < s1 - 1e-12 * abs(s1)).ravel()
            if not len(a):
                break
            y, za, qm = Y[:, a], z[a], self.qm[a]
            left = s1 - za
            ds = torch.minimum(torch.full_like(left, self.p["dz_push"]), left)
            px, py, pz = y[3], y[4], y[5]
            g = torch.sqrt(1 + px * px + py * py + pz * pz)
            lims = [0.5 * self.h * pz * (g + pz) / (1 + px * px + py * py)]
            if self.p["laser_on"]:
                hl = g - px * math.sin(self.p["theta"]) - pz * math.cos(self.p["theta"])
                lims.append(self.p["push_phase"] * pz / (self.p["kL"] * hl.clamp_min(1e-12)))
            for lim in lims:
                ds = torch.where(lim < ds, left / torch.ceil(left / lim), ds)
            k1 = self.rhs(y, za, qm)
            k2 = self.rhs(y + 0.5 * ds * k1, za + 0.5 * ds, qm)
            k3 = self.rhs(y + 0.5 * ds * k2, za + 0.5 * ds, qm)
            k4 = self.rhs(y + ds * k3, za + ds, qm)
            Y[:, a] = y + ds / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
            z[a] = za + ds
        self.q = list(Y)
        self.alive &= (self.q[2] >= 0) & (self.q[2] < float(self.c.zeta[-1]))

    # ------------------------------------------------------------ the streaming plasma
    @staticmethod
    def boris(u, E, B, qm, dt):
        qh = 0.5 * qm * dt
        m = [u[k] + qh * E[k] for k in range(3)]
        qg = qh / torch.sqrt(1 + m[0] ** 2 + m[1] ** 2 + m[2] ** 2)
        t = [qg * B[k] for k in range(3)]
        cross = lambda a, b: [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]  # noqa: E731
        c = cross(m, t)
        up = [m[k] + c[k] for k in range(3)]
        sf = 2 / (1 + t[0] ** 2 + t[1] ** 2 + t[2] ** 2)
        c = cross(up, t)
        return [m[k] + sf * c[k] + qh * E[k] for k in range(3)]

    def load_plasma(self, s0, s1):
        P = dict(configs.default_plasma(), **self.c.plasma)
        px, py, nx, ny = P["ppc_x"], P["ppc_y"], self.nx, self.ny
        A = lambda n: torch.arange(n, dtype=torch.float64, device=self.dev)  # noqa: E731
        x = ((A(nx)[:, None] + (A(px)[None, :] + 0.5) / px) * self.dx)
        y = ((A(ny)[:, None] + (A(py)[None, :] + 0.5) / py) * self.dy)
        # rows j, cells i, sub-cells b, a
        X = x[None, :, None, :].expand(ny, nx, py, px).reshape(-1)
        Y = y[:, None, :, None].expand(ny, nx, py, px).reshape(-1)
        w = P["n0"] * self.dx * self.dy * (s1 - s0) / (px * py)
        kinds = [(-1.0, -1.0, 1.0)] + [(I["Z0"], I["Z0"] / I["mass"], I["atoms"]) for I in self.c.ions]
        m = len(kinds)
        rep = lambda v: torch.tensor(v, dtype=torch.float64, device=self.dev).repeat(len(X))  # noqa: E731
        zero = torch.zeros(m * len(X), dtype=torch.float64, device=self.dev)
        self.S = dict(x=X.repeat_interleave(m), y=Y.repeat_interleave(m), z=zero + s0, u=[zero.clone() for _ in range(3)],
                      qw=rep([k[0] * k[2] * w for k in kinds]), qm=rep([k[1] for k in kinds]),
                      live=torch.ones_like(zero, dtype=torch.bool))
        self.P = P

    def stream(self, n, s1, last):
        """The particles through half-cell n with the fields of slices n and n + 1; the current [3, ny, nx]."""
        S, h, Delta = self.S, self.h, self.p["dz"]
        cut = lambda v: v[self.sel]                          # noqa: E731
        x, y, z, qw, qm = (cut(S[k]) for k in ("x", "y", "z", "qw", "qm"))
        u = [cut(v) for v in S["u"]]
        a0 = 1 + u[0] ** 2 + u[1] ** 2
        g0 = torch.sqrt(a0 + u[2] ** 2)
        omv = a0 / (g0 * (g0 + u[2]))
        dt0 = h / omv
        hd = 0.5 * dt0 / g0
        k, w = self.stencil(x + hd * u[0], y + hd * u[1])
        mid = 0.5 * (self.F[:, n] + self.F[:, n + 1]).reshape(6, -1)
        e = torch.zeros(6, len(x), dtype=torch.float64, device=self.dev)
        for s in range(9):
            e += w[s] * mid[:, k[s]]
        E, B = e[:3], e[3:]
        v1 = self.boris(u, E, B, qm, dt0)
        a1 = 1 + v1[0] ** 2 + v1[1] ** 2
        g1 = torch.sqrt(a1 + v1[2] ** 2)
        dt = 2 * h / (omv + a1 / (g1 * (g1 + v1[2])))

        def velocity(dt):
            v = self.boris(u, E, B, qm, dt)
            g = torch.sqrt(1 + v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
            return v, g, [0.5 * (u[k] / g0 + v[k] / g) for k in range(3)]
        v, g, vel = velocity(dt)
        trap = z + vel[2] * dt >= s1
        if bool(trap.any()):
            dtp = ((s1 - z) / vel[2].clamp_min(1e-3)).clamp_min(0.0)
            dt = torch.where(trap, dtp, dt)
            v, g, vel = velocity(dt)
        xn, yn = x + vel[0] * dt, y + vel[1] * dt
        k, w = self.stencil(0.5 * (x + xn), 0.5 * (y + yn))
        f = qw * dt / (Delta * h * self.dx * self.dy)
        J = torch.zeros(4, self.ny * self.nx, dtype=torch.float64, device=self.dev)
        neg = f.clamp_max(0.0)
        for s in range(9):
            for c in range(3):
                J[c].index_add_(0, k[s], f * w[s] * vel[c])
            if last:
                J[3].index_add_(0, k[s], neg * w[s])
        fast = trap & (v[2] / g >= self.P["vz_beam"])
        if bool(fast.any()):                                 # joins the beam: its beam current from now on
            k, w = self.stencil(xn[fast], yn[fast])
            vz = v[2][fast] / g[fast]
            f = qw[fast] / (h * self.dx * self.dy * vz)
            for s in range(9):
                for c in range(3):
                    J[c].index_add_(0, k[s], f * w[s] * v[c][fast] / g[fast])
                J[3].index_add_(0, k[s], f.clamp_max(0.0) * w[s])
        if last:
            i0, j0 = round(-self.X0 / self.dx) % self.nx, round(-self.Y0 / self.dy) % self.ny
            rho = J[3].view(self.ny, self.nx)
            self.lines[n, :self.nx], self.lines[n, self.nx:] = rho[j0], rho[:, i0]
            for key, val in (("x", xn), ("y", yn), ("z", z + vel[2] * dt)):
                S[key][self.sel] = val
            for c in range(3):
                S["u"][c][self.sel] = v[c]
            self.trapped = (self.trapped[0] + int(fast.sum()), self.trapped[1] + float(qw[fast].sum()))
            self.sel = self.sel[~trap]
        return J[:3].view(3, self.ny, self.nx)

    def march_plasma(self, s0, s1):
        self.load_plasma(s0, s1)
        N, D, P = self.N, 0.5 * (s1 - s0), self.P
        jk = self.jk
        filt = self.filt / (1 + P["smooth_length"] ** 2 * self.k2s)
        self.lines = torch.zeros(N, self.nx + self.ny, dtype=torch.float64, device=self.dev)
        self.sel = torch.arange(len(self.S["x"]), device=self.dev)
        self.js = torch.zeros(3, N + 1, self.ny, self.H, dtype=torch.complex128, device=self.dev)
        level = lambda n: ([self.R[0][n].clone(), self.R[1][n].clone()], self.E[n].clone(), self.B[n].clone())  # noqa: E731
        self.march_slice(N - 1, D, *level(N - 1))
        self.real(N - 1, N)
        zero = torch.zeros(3, self.ny, self.H, dtype=torch.complex128, device=self.dev)
        pin, dl = zero, None                                 # the current of level s0 is zero at the start of a run
        for n in range(N - 2, -1, -1):
            was = pin
            cur, pin = pin, zero
            old = level(n)
            for k in range(P["iterations"]):
                u = filt * torch.fft.rfft2(self.stream(n, s1, k + 1 == P["iterations"]))
                for c in range(3):
                    jk[c][n + 1] += u[c] - cur[c]
                cur = u
                if P["predictor_extrapolate"] and n >= 1:
                    t = u if dl is None else 2 * u - dl      # uniform zeta: weight 1
                    for c in range(3):
                        jk[c][n] += t[c] - pin[c]
                    pin = t
                self.march_slice(n, D, *old)
                self.real(n, n + 1)
            for c in (0, 1):
                self.R[c][n + 1] -= 0.5 * D * (cur[c] - was[c])
            self.js[:, n + 1] = cur
            dl = cur
        jk[2] = jk[2] - self.js[2]

    def step(self):
        dz = self.p["dz"]
        self.push(0.0, dz)
        if self.c.plasma is not None:
            self.currents(True)
            self.march_plasma(0.0, dz)
        else:
            self.currents(False)
            self.march(0.5 * dz)
        self.sponge_and_real()
        self.j0 = self.jk[:2]
        self.s = dz

    def sums(self):
        x, y, zeta, px, py, pz = (v[self.alive] for v in self.q)
        w = self.w[self.alive]
        on = self.p["laser_on"]
        kx, kz = (math.sin(self.p["theta"]), math.cos(self.p["theta"])) if on or self.p["theta"] else (0.0, 1.0)
        g = torch.sqrt(1 + px * px + py * py + pz * pz)
        X, Y = x + self.X0, y + self.Y0
        et = self.s - (zeta - self.p["zeta_center"]) - kx * X - kz * self.s
        v = [torch.ones_like(X), X, Y, zeta, X * X, Y * Y, zeta * zeta, px, py, pz, g, px * kx + pz * kz, pz * pz, et]
        wl = torch.full((self.N,), self.h, dtype=torch.float64, device=self.dev)
        wl[0] = wl[-1] = 0.5 * self.h
        en = sum(float((wl * (self.F[c, :self.N] ** 2).sum(dim=(1, 2))).sum()) for c in range(6))
        S = [float((w * t).sum()) for t in v] + [float(len(w)), 0.5 * self.dx * self.dy * en, float((~self.alive).sum()),
                                                 float(self.trapped[0]), self.trapped[1]]
        return np.array(S)


def exact(case, seed):
    # gas: the event set hangs on a random sequence; adjoint: hours of steps to differentiate in this form
    if case["kind"] in ("gas", "adjoint"):
        return None
    cfg, parts = inputs(case, seed)
    m = _March(cfg, parts)
    m.start()
    m.step()
    out = {"sums": m.sums(), "F": m.F}
    if case["kind"] == "exchange":
        out.update({f: v.cpu().numpy() for f, v in zip(("x", "y", "zeta", "px", "py", "pz"), m.q)})
        return out
    pair = torch.view_as_real
    out.update(Rx=pair(m.R[0]), Ry=pair(m.R[1]), j0x=pair(m.j0[0].contiguous()), j0y=pair(m.j0[1].contiguous()))
    if cfg.plasma is not None:
        # mixed: the density on the axis hangs on single trapped electrons there, a realisation and no value
        out["rho_lines"] = m.lines if case["form"] == "fp64" else None
    else:
        out["jkz"] = pair(m.jk[2].contiguous())
    return out
