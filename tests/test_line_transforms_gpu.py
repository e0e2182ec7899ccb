"""The kernels that work on whole lines of the window (rows of the currents, of the sponge and of the real fields, columns,
the march, the push with its held stencil) at every transform length and at the ends of their ranges, against the numpy
restatement of the march (oracle/g3d_oracle.py), and the field energy against its sum over F.

Tolerances: FP64 spectra <= 1e-10 of the field state norm and particles <= 1e-10 as in test_parity_gpu.py, the float F <= 1e-6,
the mixed form <= 1e-5 (test_mixed_gpu.py).
"""
import numpy as np
import pytest

from conftest import CURRENTS, FIELDS, assert_state, rel_l2, state_errors
from g3d_oracle import Oracle

pytestmark = pytest.mark.gpu

# every length along x and along y, few slices (down to the shortest window, fewer than the march streams ahead)
SIZES = [(8, 4, 4), (8, 512, 5), (16, 8, 7), (24, 48, 9), (32, 24, 12), (48, 32, 10), (64, 96, 11), (96, 64, 13), (128, 192, 6),
         (192, 128, 6), (256, 16, 9), (384, 16, 5), (512, 8, 6), (16, 384, 5), (64, 256, 8)]


def run(cfg, precision="fp64", steps=1):
    from g3d import Simulation
    s = Simulation(cfg, precision=precision)
    s.load_bunch()
    o = Oracle(cfg)
    o.set_particles(s.host_particles())
    o.set_origin(s.status().X0, s.status().Y0)
    s.init_fields()
    o.init_fields()
    for _ in range(steps):
        s.step()
        o.step()
    return s, o


@pytest.mark.parametrize("nx,ny,nz", SIZES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_step_at_every_transform_length(nx, ny, nz, precision):
    from g3d import configs
    cfg = configs.config2(nx=nx, ny=ny, nzeta=nz, nmacro=3000, steps=1)       # sponge, k filters, the plane wave
    s, o = run(cfg, precision)
    try:
        got, ref = {a: s.array(a) for a in FIELDS + CURRENTS}, {a: o.array(a) for a in FIELDS + CURRENTS}
        if precision == "fp64":
            assert_state(got, ref, FIELDS, 1e-10, comp_tol=1e-5)
            assert_state(got, ref, CURRENTS, 1e-10, comp_tol=1e-5)
            assert rel_l2(s.array("F"), o.array("F")) <= 1e-6
        else:
            for names in (FIELDS, CURRENTS):
                assert max(e for e, _ in state_errors(got, ref, names).values()) <= 1e-5
            assert rel_l2(s.array("F"), o.array("F")) <= 1e-5
        p, q = s.host_particles(), o.host_particles()
        for f in ("x", "y", "zeta", "px", "py", "pz"):
            assert rel_l2(p[f], q[f]) <= (1e-10 if precision == "fp64" else 1e-6), f
    finally:
        s.close()


@pytest.mark.parametrize("zeta_filter,graded", [(0, False), (1, False), (1, True)])
def test_push_through_many_cells_and_slices(zeta_filter, graded):
    """Slow particles over long steps: every sub-step starts in another cell or half-cell than the one before, so the
    stencil held in shared memory has to be loaded anew, and some particles leave the window. On a graded axis the held
    half-cell is also what locates them."""
    from g3d import configs
    cfg = configs.config1(nx=32, ny=16, nzeta=24, nmacro=5000, steps=1)
    cfg.bunches[0].update(gamma=4.0, emitx=2.0, emity=2.0, sigz=8.0, zeta_center=20.0)
    cfg.params.update(dz=12.0, dz_push=0.7, zeta_filter=zeta_filter)
    if graded:
        configs.on_graded_zeta(cfg)
    s, o = run(cfg, steps=2)
    try:
        p, q = s.host_particles(), o.host_particles()
        assert np.array_equal(p["alive"], q["alive"]) and 0 < np.count_nonzero(q["alive"] != 1) < len(q)
        a = q["alive"] == 1
        for f in ("x", "y", "zeta", "px", "py", "pz"):
            # the float F of both codes differs by its last bit here and there (1e-8), which the strong self fields of a
            # slow bunch carry into the momenta
            assert rel_l2(p[f][a], q[f][a]) <= 1e-8, f
    finally:
        s.close()


@pytest.mark.parametrize("build", ["fourier", "odd rows between walls", "graded"])
def test_field_energy_is_the_sum_over_the_dual_cells(build):
    from g3d import Simulation, configs
    if build == "fourier":
        cfg = configs.config1(nx=24, ny=8, nzeta=37, nmacro=4000, steps=1)
    elif build == "graded":
        cfg = configs.on_graded_zeta(configs.config1(nx=16, ny=16, nzeta=64, nmacro=4000, steps=1))
    else:
        cfg = configs.freehand_small(half=12)
        cfg.ynode = cfg.ynode[:-1]                       # 23 cells: an odd number of rows
        cfg.ny = 23
        cfg.Ly = float(cfg.ynode[-1] - cfg.ynode[0])
    s = Simulation(cfg)
    try:
        s.init()
        s.step()
        F = s.array("F").reshape(6, cfg.nzeta + 2, cfg.ny, cfg.nx)[:, :cfg.nzeta].astype(np.float64)
        h = np.diff(cfg.zeta)
        wl = 0.5 * (np.concatenate([[0.0], h]) + np.concatenate([h, [0.0]]))
        if cfg.ynode is None:
            node = half = np.full(cfg.ny, cfg.Ly / cfg.ny)
        else:
            cell = np.diff(cfg.ynode)
            half = cell
            node = np.concatenate([[cell[0]], 0.5 * (cell[1:] + cell[:-1])])
        e = sum(0.5 * np.einsum("l,j,lji->", wl, half if c in (1, 3, 5) else node, F[c] ** 2) for c in range(6)) * cfg.Lx / cfg.nx
        # the wall row (j = 0) of the node components is zero, whatever its dual cell
        assert abs(s.field_energy() - e) <= 1e-12 * e
    finally:
        s.close()
