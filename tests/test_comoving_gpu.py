"""The co-moving start field's solves along zeta against the numpy restatement (oracle/g3d_oracle.py): the parallel reduction
from the shortest window to its longest, the sweep just above it and above the modes up to which the reduction is faster, and
the pointwise solve of beta = 1 that the whole start makes after them.

Tolerance: the rows are diagonally dominant by k_perp^2, so neither elimination order amplifies its rounding: FP64 <= 1e-11
of the state norm (1e-10 after the relaxation's marches), the mixed form's float j_z <= 1e-6.
"""
import numpy as np
import pytest

from conftest import rel_l2, state_errors
from g3d_oracle import Oracle

pytestmark = pytest.mark.gpu


NARROW = [(16, 8, nz) for nz in (4, 5, 255, 256, 257, 1025, 3200, 3201)]
WIDE = [(192, 192, 6), (256, 192, 6), (384, 192, 6), (384, 256, 5)]       # 18,624, 24,768, 37,056 and 49,408 modes


def sweep(nx, ny, nz, precision):
    """The rule of the dispatch (pcr_modes, csrc/k_comoving.cuh)."""
    f32 = precision == "mixed"
    line = 0 if nz > 3200 else (40000 if f32 else 20000) if nz <= 1024 else (20000 if f32 else 13000)
    return ny * (nx // 2 + 1) > line


@pytest.mark.parametrize("nx,ny,nz", NARROW + WIDE)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_start_field(nx, ny, nz, precision):
    from g3d import Simulation, configs
    cfg = configs.config1(nx=nx, ny=ny, nzeta=nz, nmacro=3000, steps=1)
    cfg.bunches[0].update(gamma=1.5, emitx=0.0, emity=0.0)              # gamma^-2 far from 0: the off-diagonals matter
    s = Simulation(cfg, precision=precision)
    try:
        s.load_bunch()
        o = Oracle(cfg)
        o.set_particles(s.host_particles())
        o.set_origin(s.status().X0, s.status().Y0)
        s.currents(); o.currents()
        s.profile(True)
        s.comoving_field(); o.comoving_field()
        assert ("comoving_sweep" in s.profile_results()) == sweep(nx, ny, nz, precision)
        s.profile(False)
        for a in ("Rx", "Ry"):
            assert np.linalg.norm(o.array(a)) > 0
            assert rel_l2(s.array(a), o.array(a)) <= (1e-11 if precision == "fp64" else 1e-6), a
        s.init_fields(); o.init_fields()
        names = ("Rx", "Ry")
        e = state_errors({a: s.array(a) for a in names}, {a: o.array(a) for a in names}, names)
        assert max(v for v, _ in e.values()) <= (1e-10 if precision == "fp64" else 1e-6)
    finally:
        s.close()
