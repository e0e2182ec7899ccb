"""The slice loop of the streaming plasma on the Fourier y grid (push, rows, columns with the slice march and the half-cell's
correction, rows of the real fields) against the 64-bit restatement of a step that perf/cases.py holds: one s-step from the
start field over transform lengths along x and y, pass counts, predictors of one and several passes, species, smoothing, both
forms. Tolerances: those stated with the restatement (four times the distance that the float F leaves), per output.
"""
import importlib.util
import os

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cases():
    cwd = os.getcwd()
    os.chdir(REPO)
    try:
        spec = importlib.util.spec_from_file_location("measured_cases", os.path.join(REPO, "perf", "cases.py"))
        m = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(m)
        return m
    finally:
        os.chdir(cwd)


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny,nz,ppc,ions,passes,smooth", [
    (16, 16, 100, 1, False, 1, 0.0), (16, 256, 80, 1, True, 2, 0.0), (256, 16, 80, 1, True, 2, 0.4), (24, 96, 90, 2, True, 3, 0.0),
    (96, 24, 90, 1, False, 2, 0.0), (48, 192, 70, 1, True, 1, 0.4), (512, 16, 70, 1, False, 2, 0.0), (16, 512, 70, 1, True, 2, 0.0),
    (384, 32, 70, 1, False, 2, 0.0), (32, 4, 70, 2, True, 2, 0.0), (8, 32, 70, 2, True, 2, 0.0)])
def test_step_matches_the_restatement(cases, form, nx, ny, nz, ppc, ions, passes, smooth):
    import torch
    case = dict(kind="lwfa", nx=nx, ny=ny, nz=nz, n=2000, form=form, ppc=ppc, ions=ions, passes=passes, smooth=smooth)
    state = cases.prepare(case, 3)
    got, want = cases.run(state), cases.exact(case, 3)
    tol = cases.tolerance(case)["rel"]
    for name, w in want.items():
        if w is None:
            continue
        g, w = torch.as_tensor(got[name]).double().cpu().ravel(), torch.as_tensor(w).double().cpu().ravel()
        assert float((g - w).norm()) <= tol * float(w.norm()), name
    state["sim"].close()


def test_graph_and_direct_launches_agree(cases):
    """The first two marches with a set of buffers are launched kernel by kernel, later ones as the captured graph; with the
    kernels timed one by one every march is launched directly. All give the same run up to the order of the adds."""
    case = dict(kind="lwfa", nx=32, ny=32, nz=100, n=2000, form="fp64", ppc=2, ions=True, passes=2, smooth=0.0)
    out = []
    for profiled in (False, True):
        state = cases.prepare(case, 3)
        state["sim"].profile(profiled)
        for _ in range(6):
            cases.run(state)
        assert state["sim"].graph_count() == (0 if profiled else 2)      # two sets of buffers take turns: steps 5 and 6
        out.append({a: state["sim"].array(a) for a in ("Rx", "Ry", "Ez", "F")})
        state["sim"].close()
    for a in out[0]:
        d, n = np.linalg.norm(out[0][a] - out[1][a]), np.linalg.norm(out[1][a])
        assert d <= 1e-8 * n, (a, d / n)       # six steps amplify the adds' rounding (1e-16) by the wake's growth


@pytest.mark.parametrize("nx,half,form,graph", [(16, 12, "fp64", True), (64, 32, "fp64", True), (64, 32, "mixed", True),
                                                (256, 64, "mixed", False), (48, None, "fp64", False), (32, None, "mixed", True)])
def test_small_grids_march_as_a_graph(nx, half, form, graph):
    """Which grids' slice loop becomes a graph (GRAPH_POINTS in csrc/g3d_plasma.cu): the free-hand grid's loop has twice the
    launches and is bound by them up to larger grids."""
    from g3d import Simulation, configs
    cfg = configs.lwfa_small(nx=nx, ny=nx, nzeta=24, nmacro=500, steps=6, ppc=1)
    if half:
        configs.on_freehand_y(cfg, half=half, grow=1.03)
    s = Simulation(cfg, precision=form)
    try:
        s.init()
        for _ in range(6):
            s.step()
        assert (s.graph_count() > 0) == graph
        assert np.isfinite(s.array("Ez")).all()
    finally:
        s.close()
