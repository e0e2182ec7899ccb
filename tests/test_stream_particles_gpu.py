"""The streaming particles of the plasma march without the reference: the deposit on the free-hand y grid (a warp's particles with
equal stencils summed first) against a CPU sum over the particles' straight paths, some of them at and beyond the walls; field
ionization of fixed and of mobile ions on both y grids against the host's rates, random numbers and gathers; the density
lines of particles at rest. Densities so low that no particle acts on a field make all of these exact.

Tolerances: FP64 sums of some hundred terms <= 1e-12, the mixed form's FP32 planes 1e-6; the density lines are FP64 sums in both
forms on the free-hand grid, of FP32 charges (2^-24, with FP32 weights 2e-6) in the mixed form on the Fourier grid. Events: exact, but
for an ion whose waiting time is closer to the time left than the float F can tell (the rate's logarithm moves by some thirty
times F's 1e-7, 1e-6 in the mixed form).
"""
import math

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


# ---------------------------------------------------------------- grids
def locate(X, v):
    """The axis' node index and fraction, the end cells continued beyond the ends."""
    n = len(X)
    i = np.clip(np.searchsorted(X, v, side="right") - 1, 0, n - 2)
    t = i + (v - X[i]) / (X[i + 1] - X[i])
    return np.where(v >= X[-1], n - 1 + (v - X[-1]) / (X[-1] - X[-2]), t)


def tsc(t):
    c = np.floor(t + 0.5)
    f = t - c
    return c.astype(int), np.stack([0.5 * (0.5 - f) ** 2, 0.75 - f * f, 0.5 * (0.5 + f) ** 2])


class Grid:
    """TSC stencils of points (x in the box, y) and the inverse dual cells of a configuration."""

    def __init__(self, cfg):
        self.nx, self.ny, self.dx = cfg.nx, cfg.ny, cfg.Lx / cfg.nx
        self.walls = cfg.ynode is not None
        if self.walls:
            self.yn = np.asarray(cfg.ynode)
            cell = np.diff(self.yn)
            self.iD = 1 / cell
            self.iA = 1 / np.concatenate([[cell[0]], 0.5 * (cell[1:] + cell[:-1])])
        else:
            self.dy = cfg.Ly / cfg.ny
            self.iD = self.iA = np.full(cfg.ny, 1 / self.dy)

    def points(self, x, y, half):
        """(rows [3, n], columns [3, n], weights of both); rows beyond the walls are out of range."""
        cx, wx = tsc(x / self.dx)
        cy, wy = tsc((locate(self.yn, y) if self.walls else y / self.dy) - (0.5 if half and self.walls else 0.0))
        o = np.arange(-1, 2)[:, None]
        rows = cy[None] + o
        return (rows if self.walls else rows % self.ny), (cx[None] + o) % self.nx, wy, wx

    def add(self, plane, x, y, f, half):
        r, c, wy, wx = self.points(x, y, half)
        lo = 0 if half or not self.walls else 1              # the wall row of the nodes takes nothing
        inv = self.iD if half else self.iA
        for v in range(3):
            ok = (r[v] >= lo) & (r[v] < self.ny)
            for u in range(3):
                np.add.at(plane, (r[v][ok], c[u][ok]), (f * wy[v] * wx[u])[ok] * inv[r[v][ok]])

    def gather(self, plane, x, y, half):
        r, c, wy, wx = self.points(x, y, half)
        out = np.zeros(len(x))
        for v in range(3):
            ok = (r[v] >= 0) & (r[v] < self.ny)
            for u in range(3):
                out[ok] += (wy[v] * wx[u])[ok] * plane[r[v][ok], c[u][ok]]
        return out

    def lines(self, plane, i0, j0):
        return np.concatenate([plane[j0], plane[:, i0]])


def axis_cell(cfg, st):
    dx = cfg.Lx / cfg.nx
    j0 = cfg.ny // 2 if cfg.ynode is not None else round(-st.Y0 / (cfg.Ly / cfg.ny)) % cfg.ny
    return round(-st.X0 / dx) % cfg.nx, j0


# ---------------------------------------------------------------- deposit between walls
@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("n,passes", [(33, 1), (700, 2)])
def test_deposit_between_walls_is_the_sum_over_the_paths(form, n, passes):
    from g3d import PARTICLE_DTYPE, Simulation, configs
    cfg = configs.freehand_small(nx=16, half=9, nzeta=13, steps=1, sponge=0.0, zeta_filter=0, k_filter=0)
    cfg.bunches = []
    cfg.params.update(dz=60.0, dz_push=60.0, z_end=60.0)         # nobody is trapped: z advances by less
    cfg.plasma = dict(n0=1e-9, r_max=1e-9, iterations=passes, ppc_x=1, ppc_y=1)   # the lattice is empty
    cfg.ions = [configs.ion_species("H", 1, 1.0)]                # (a species, so that positive charge has lines)
    rng = np.random.default_rng(n)
    yn = np.asarray(cfg.ynode)
    p = np.zeros(n, dtype=PARTICLE_DTYPE)
    p["x"], p["zeta"] = rng.uniform(0, cfg.Lx, n), rng.uniform(0.3, cfg.zeta[-1], n)
    p["y"] = rng.uniform(yn[0], yn[-1], n)                       # the cells at the walls among them
    p["y"][: n // 4] = yn[1] + 0.02 * rng.standard_normal(n // 4)
    p["y"][n // 4: n // 3] = yn[-2] + 0.02 * rng.standard_normal(n // 3 - n // 4)
    p["x"][n // 2:] = p["x"][: n - n // 2]                       # shared stencils: the same (x, y) and neighbours
    p["y"][n // 2:] = p["y"][: n - n // 2] + 1e-3 * rng.standard_normal(n - n // 2)
    p["px"], p["py"], p["pz"] = 0.6 * rng.standard_normal(n), 0.6 * rng.standard_normal(n), rng.uniform(-0.4, 0.4, n)
    p["py"][::9] *= 40
    p["y"][0], p["py"][0], p["y"][1], p["py"][1] = yn[0] + 0.03, -30, yn[-1] - 0.03, 30     # the middle of the path beyond a wall
    p["w"], p["q"] = 1e-16 * rng.uniform(0.5, 1.5, n), rng.choice([-1.0, 1.0], n)
    p["qm"], p["alive"], p["id"] = p["q"], 1, np.arange(n)

    s = Simulation(cfg, precision=form)
    try:
        s.init_fields()
        s.set_particles(p)
        s.step()                                                 # all slower than vz_min: they stream in this march
        st = s.status()
        got = [s.array(a).reshape(cfg.nzeta + 1, cfg.ny, cfg.nx)[1:-1] for a in ("j0x", "j0y")]
        lines = [s.array(a).reshape(cfg.nzeta, -1) for a in ("rho_lines", "rho_lines_i")]
        end = s.streaming_particles()
    finally:
        s.close()

    g = Grid(cfg)
    i0, j0 = axis_cell(cfg, st)
    ga = np.sqrt(1 + p["px"] ** 2 + p["py"] ** 2 + p["pz"] ** 2)
    v = np.stack([p["px"] / ga, p["py"] / ga, p["pz"] / ga])
    x, y, zeta, on = p["x"].copy(), p["y"].copy(), p["zeta"].copy(), np.ones(n, bool)
    z = np.asarray(cfg.zeta)
    J = np.zeros((2, cfg.nzeta - 1, cfg.ny, cfg.nx))
    rho = np.zeros((2, cfg.nzeta, cfg.ny, cfg.nx))
    beyond = 0
    for m in range(cfg.nzeta - 2, -1, -1):
        h = z[m + 1] - z[m]
        k = np.flatnonzero(on & (zeta > z[m]))
        hl = np.where(zeta[k] >= z[m + 1] - 1e-9 * h, h, zeta[k] - z[m])
        dt = hl / (1 - v[2, k])
        xn, yn1 = x[k] + v[0, k] * dt, y[k] + v[1, k] * dt
        f = p["q"][k] * p["w"][k] * dt / (60.0 * h * g.dx)
        xm, ym = (0.5 * (x[k] + xn)) % cfg.Lx, 0.5 * (y[k] + yn1)
        g.add(J[0, m], xm, ym, f * v[0, k], False)
        g.add(J[1, m], xm, ym, f * v[1, k], True)
        for c, sgn in enumerate((f < 0, f > 0)):
            g.add(rho[c, m], xm[sgn], ym[sgn], f[sgn], False)
        beyond += np.count_nonzero((ym < yn[0]) | (ym > yn[-1]))
        x[k], y[k], zeta[k] = xn, yn1, z[m]
        on[k[(yn1 < yn[1]) | (yn1 > yn[-2])]] = False
    assert beyond > 0 and 0 < np.count_nonzero(on) < n
    assert np.array_equal(end["alive"] == 0, ~on)
    tol = 1e-12 if form == "fp64" else 1e-6
    for c in range(2):
        want = np.fft.fft(J[c], axis=2)
        want[:, :, cfg.nx // 2] = 0                              # the Nyquist mode is not kept
        assert rel_l2(got[c], want) <= tol, c
        assert rel_l2(lines[c], np.stack([g.lines(r, i0, j0) for r in rho[c]])) <= 1e-12, c


# ---------------------------------------------------------------- ionization
M64 = (1 << 64) - 1


def mix64(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


def adk(cfg, sp, zmax):
    """(ln prefactor, power, exponent, peak) per level in code units: the s-state ADK rate, over omega_0, of E / E_0."""
    c, me, e = 2.99792458e8, 9.1093837015e-31, 1.602176634e-19
    wa, Ea, UH = 4.1341373335e16, 5.14220674763e11, 13.605693122994       # atomic frequency [1/s] and field [V/m], Rydberg [eV]
    w0 = 2 * math.pi * c / cfg.params["lambda0"]
    E0 = me * c * w0 / e
    out = []
    for k in range(zmax):
        x = sp["ip_eV"][k] / UH
        ns = (k + 1) / math.sqrt(x)
        power = 2 * ns - 1
        pre = (math.log(wa) + 2 * ns * math.log(2) - math.log(ns) - math.lgamma(ns + 1) - math.lgamma(ns) + math.log(0.5 * x)
               + power * math.log(2 * x ** 1.5 * Ea))
        expo = -(2 / 3) * x ** 1.5 * Ea / E0
        out.append((pre - math.log(w0) - power * math.log(E0), power, expo, -expo / power if power > 0 else 1e300))
    return out


def rate(L, E):
    if not E > 0:
        return 0.0
    E = min(E, L[3])
    return math.exp(L[0] - L[1] * math.log(E) + L[2] / E)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("walls", [False, True], ids=["fourier", "walls"])
@pytest.mark.parametrize("mobile", [False, True], ids=["fixed", "mobile"])
def test_ionization_events_and_charge_lines(form, walls, mobile):
    from g3d import Simulation, configs
    cfg = configs.ionization_small()
    cfg.ions = [configs.ion_species("H", 0, 1.0, ionization=True, mobile=mobile),
                configs.ion_species("N", 1, 1.0, ionization=True, mobile=mobile)]        # N enters singly charged
    for i in cfg.ions:
        i["mass"] = 1e15                                         # a mobile ion's push runs, but does not carry it anywhere
    cfg.plasma["n0"] = 1e-13
    cfg.params.update(sponge=0.0, sponge_y=0.0)
    if walls:
        configs.on_freehand_y(cfg)
    s = Simulation(cfg, precision=form)
    try:
        s.init()
        s.step()
        st = s.status()
        F = s.array("F").reshape(6, cfg.nzeta + 2, cfg.ny, cfg.nx).astype(np.float64)
        q = s.streaming_particles()
        lines = s.array("rho_lines_i").reshape(cfg.nzeta, -1)
        nfreed = int(np.count_nonzero((q["sp"] >= 50) & (q["sp"] < 100)))
    finally:
        s.close()
    ion = q[(q["sp"] >= 3) & (q["sp"] < 50)]
    assert len(ion) == 2 * (cfg.nx * (cfg.ny - (2 if walls else 0)))
    g = Grid(cfg)
    i0, j0 = axis_cell(cfg, st)
    z = np.asarray(cfg.zeta)
    lev = [adk(cfg, sp, sp["Zmax"]) for sp in cfg.ions]
    step = mix64((cfg.plasma["seed"] * 0x9E3779B97F4A7C15 + st.istep) & M64)
    x, y = ion["x"], ion["y"]
    Z = np.array([cfg.ions[k - 3]["Z0"] for k in ion["sp"]])
    sure = np.ones(len(ion), bool)
    freed = 0
    rho = np.zeros((cfg.nzeta, cfg.ny, cfg.nx))
    eps = 1e-4 if form == "fp64" else 1e-3
    E = [np.sqrt(sum(g.gather(F[c, n], x, y, c == 1) ** 2 for c in range(3))) for n in range(cfg.nzeta)]
    for n in range(cfg.nzeta - 2, -1, -1):
        h = z[n + 1] - z[n]
        g.add(rho[n], x, y, Z * ion["w"] * h / (cfg.params["dz"] * h * g.dx), False)
        key = mix64(step ^ ((n << 8) | (cfg.plasma.get("iterations", 2) - 1)))
        for i in np.flatnonzero(np.maximum(E[n], E[n + 1]) > 1e-3):
            L = lev[ion["sp"][i] - 3]
            base, draw, left = mix64(key ^ mix64(int(ion["id"][i]))), 0, h
            while Z[i] < len(L):
                w = 0.5 * (rate(L[Z[i]], E[n + 1][i]) + rate(L[Z[i]], E[n][i]))
                if w * h < 1e-9:
                    break
                tw = -math.log(1 - (mix64((base + draw) & M64) >> 11) * 2.0 ** -53) / w
                draw += 1
                sure[i] &= abs(tw - left) > eps * tw
                if tw > left:
                    break
                left -= tw
                Z[i] += 1
                freed += 1
    assert np.count_nonzero(~sure) <= 0.05 * len(ion)
    assert np.array_equal(ion["q"][sure], Z[sure]), (ion["q"][sure] != Z[sure]).sum()
    assert freed > 200 and abs(freed - nfreed) <= 7 * np.count_nonzero(~sure)
    assert (ion["q"] == [cfg.ions[k - 3]["Z0"] for k in ion["sp"]]).any() and (ion["q"] > 2).any()   # none, and several levels
    if sure.all():
        tol = 2e-6 if form == "mixed" and not walls and mobile else 1e-12
        assert rel_l2(lines, np.stack([g.lines(r, i0, j0) for r in rho])) <= tol


@pytest.mark.parametrize("form", ["fp64", "mixed"])
def test_charge_lines_of_particles_at_rest(form):
    """Electrons and mobile ions that do not ionize (fixed ones are not loaded), on the Fourier y grid."""
    from g3d import Simulation, configs
    cfg = configs.lwfa_small(nx=24, ny=16, nzeta=40, nmacro=500, steps=1, n0=1e-12)
    cfg.bunches, cfg.glasers = [], []
    cfg.params.update(sponge=0.0, sponge_y=0.0)
    s = Simulation(cfg, precision=form)
    try:
        s.init()
        s.step()
        st = s.status()
        q = s.streaming_particles()
        lines = [s.array(a).reshape(cfg.nzeta, -1) for a in ("rho_lines", "rho_lines_i")]
    finally:
        s.close()
    g = Grid(cfg)
    i0, j0 = axis_cell(cfg, st)
    for sp, sgn, got in ((2, -1.0, lines[0]), (3, 1.0, lines[1])):
        p = q[q["sp"] == sp]
        assert len(p) == cfg.nx * cfg.ny * 4
        plane = np.zeros((cfg.ny, cfg.nx))
        g.add(plane, p["x"] % cfg.Lx, p["y"] % cfg.Ly, sgn * p["w"] / (cfg.params["dz"] * g.dx), False)
        want = np.tile(g.lines(plane, i0, j0), (cfg.nzeta - 1, 1))
        assert rel_l2(got[:-1], want) <= (2e-6 if form == "mixed" else 1e-12), sp
        assert not got[-1].any()
