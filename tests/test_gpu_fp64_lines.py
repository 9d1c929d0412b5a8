"""The IEEE-FP64 line kernels take a direction's three RK stages in one launch
(grids whose rows and columns fit a CTA): lengths at the edges of warps, runs
and lines per CTA, against the oracle's time steps, halos and state_tmp
included; the recorded stages against the single-stage kernels; graph capture."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.solve import evolve, reset_direction
from tests.helpers import BACKGROUNDS, make_params, normwise

pytestmark = pytest.mark.gpu

# 3 steps are 18 stages of at most 3e-14 of max|s| each (test_gpu_fp64_runs.py): 6e-13.
TOL = 1e-12
GRIDS = [(2, 1), (3, 2), (4, 3), (30, 29), (31, 30), (29, 31), (60, 61), (62, 60), (63, 62), (64, 64), (100, 50),
         (124, 31), (125, 63), (481, 37), (37, 481), (480, 240), (511, 257), (991, 20), (20, 992), (992, 5), (993, 4),
         (200, 100), (256, 128), (401, 199), (512, 256), (24, 2000), (2000, 24), (3001, 40), (5, 9000), (640, 600)]


def developed(p, seed):
    f = initialize_fields(p)
    init(f, p)
    rng = np.random.default_rng(seed)
    noise = rng.standard_normal(f.shape) * np.array([1e-3, 5.0, 2.0, 0.5])[:, None, None]
    f.state += torch.from_numpy(noise).to(f.device)
    f.state_tmp.copy_(f.state + 0.5)
    return f


@pytest.mark.parametrize("nx,nz", GRIDS)
@pytest.mark.parametrize("ic,reverse", [("collision", False), ("gravity", True)])
def test_steps_vs_oracle(ic, reverse, nx, nz):
    p = make_params(nx, nz, ic)
    f = developed(p, nx * 1000 + nz)
    o = O.OracleSim(O.make_params(nx, nz, ic))
    for name in BACKGROUNDS:
        getattr(o, name)[:] = getattr(f, name).cpu().numpy()
    o.state[:], o.state_tmp[:], o.reverse = f.state.cpu().numpy(), f.state_tmp.cpu().numpy(), int(reverse)
    if f.src_w is not None:
        o.src_w[:] = f.src_w.cpu().numpy()
    reset_direction(reverse)
    evolve(p, f, None, dt=p["dt"], nsteps=1)
    evolve(p, f, None, dt=p["dt"], nsteps=2)
    reset_direction()
    o.evolve(3)
    assert max(normwise(f.state.cpu().numpy(), o.state, interior=False)) <= TOL
    assert max(normwise(f.state_tmp.cpu().numpy(), o.state_tmp, interior=False)) <= TOL


@pytest.mark.parametrize("nx,nz", [(2, 1), (31, 30), (100, 50), (63, 125), (512, 256)])
def test_no_halo_writes_and_split_calls(nx, nz):
    """step_flags 0 leaves every halo cell alone; n steps in one call and one by one give the same bits."""
    p = dict(make_params(nx, nz, "collision"), step_flags=0)
    a, b = developed(p, 5), developed(p, 5)
    ref = a.state.clone(), a.state_tmp.clone()
    reset_direction()
    evolve(p, a, None, dt=p["dt"], nsteps=4)
    reset_direction()
    for _ in range(4):
        evolve(p, b, None, dt=p["dt"])
    for got, old in ((a.state, ref[0]), (a.state_tmp, ref[1])):
        halo = torch.ones_like(got, dtype=torch.bool)
        halo[:, 2:-2, 2:-2] = False
        assert torch.equal(got[halo], old[halo])
    assert torch.equal(a.state, b.state) and torch.equal(a.state_tmp, b.state_tmp)


@pytest.mark.parametrize("nx,nz", [(3, 2), (62, 33), (250, 125)])
@pytest.mark.parametrize("reverse", (0, 1))
def test_recorded_stages_vs_stage_kernels(nx, nz, reverse):
    p = make_params(nx, nz, "gravity")
    f = developed(p, 9)
    n = f.state.numel()
    stages, end = torch.zeros(6 * n, dtype=torch.float64, device="cuda"), torch.zeros_like(f.state)
    bg = [_native.ptr(a) for a in f.backgrounds()]
    _native.call("mw_step_record_f64", nx, nz, p["dx"], p["dz"], p["dt"], p["dt"], *bg, _native.ptr(f.src_w),
                 _native.ptr(f.state), _native.ptr(stages), _native.ptr(end), reverse, 2, _native.stream_handle())
    got = [s.view(f.shape) for s in stages.split(n)] + [end]
    s = f.state.clone()
    for k in range(6):
        d = (0 if reverse else 1) if k < 3 else (1 if reverse else 0)
        base = got[0] if k < 3 else got[3]
        out = torch.zeros_like(s)
        _native.call("mw_dirstage_f64", nx, nz, p["dx"], p["dz"], p["dt"], *bg, _native.ptr(f.src_w), _native.ptr(base),
                     _native.ptr(got[k]), _native.ptr(out), p["dt"] / (3 - k % 3), d, 2, 0, _native.stream_handle())
        assert max(normwise(got[k + 1].cpu().numpy(), out.cpu().numpy())) <= TOL, k


def test_steps_under_graph_capture():
    """The launches of a call overlap (programmatic dependence); captured and replayed they give the eager bits."""
    p = make_params(100, 50, "thermal")
    a, b = developed(p, 3), developed(p, 3)
    start = a.state.clone(), a.state_tmp.clone()
    reset_direction()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        evolve(p, a, None, dt=p["dt"], nsteps=2)
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        evolve(p, a, None, dt=p["dt"], nsteps=2)
    a.state.copy_(start[0])
    a.state_tmp.copy_(start[1])
    for _ in range(3):
        g.replay()
    reset_direction()
    evolve(p, b, None, dt=p["dt"], nsteps=6)
    torch.cuda.synchronize()
    assert torch.equal(a.state, b.state) and torch.equal(a.state_tmp, b.state_tmp)


def test_noalloc_step_on_a_line_grid():
    p = make_params(120, 70, "collision")
    a, b = developed(p, 4), developed(p, 4)
    rv = ctypes.c_int(0)
    _native.call("mw_step_f64_noalloc", 120, 70, p["dx"], p["dz"], p["dt"], p["dt"],
                 *[_native.ptr(t) for t in a.backgrounds()], None, _native.ptr(a.state), _native.ptr(a.state_tmp), 3,
                 ctypes.byref(rv), 2, 1, _native.stream_handle())
    reset_direction()
    evolve(p, b, None, dt=p["dt"], nsteps=3)
    assert rv.value == 1 and torch.equal(a.state, b.state) and torch.equal(a.state_tmp, b.state_tmp)
