"""The double-FP32 line kernels take a direction's three RK stages in one
launch (grids whose rows and columns fit a CTA): lengths at the edges of warps,
runs and lines per CTA, against the oracle's time steps, halos and state_tmp
included; the recorded stages against the single-stage kernels; the latter's
64-bit-index instance; graph capture.

Tolerance of a stage: pair operations are good to 2^-47 of their operands, and
a stage's increment, dt / (12 d) times a difference of two fluxes that are sums
of at most 8 such terms and the interpolations' 16 units, stays below max|s|
(the CFL limit): 2 x 24 x 2^-47 = 3.4e-13 of max|s|; 18 stages of 3 steps 6e-12."""
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

TOL_STAGE, TOL = 1e-12, 1e-11
GRIDS = [(2, 1), (3, 2), (4, 3), (31, 30), (32, 31), (33, 32), (30, 62), (62, 63), (63, 64), (100, 50), (124, 31),
         (481, 37), (37, 481), (480, 240), (621, 20), (20, 621), (992, 5), (200, 100), (256, 128), (401, 199),
         (512, 256), (24, 2000), (2000, 24), (3001, 40), (5, 9000), (900, 600), (1000, 581)]


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
    p = dict(make_params(nx, nz, ic), f64_mode="split")
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


@pytest.mark.parametrize("nx,nz", [(2, 1), (32, 31), (100, 50), (512, 256)])
def test_no_halo_writes_and_split_calls(nx, nz):
    """step_flags 0 leaves every halo cell alone; n steps in one call and one by one give the same bits."""
    p = dict(make_params(nx, nz, "collision"), step_flags=0, f64_mode="split")
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
                 _native.ptr(f.state), _native.ptr(stages), _native.ptr(end), reverse, 1, _native.stream_handle())
    got = [s.view(f.shape) for s in stages.split(n)] + [end]
    for k in range(6):
        d = (0 if reverse else 1) if k < 3 else (1 if reverse else 0)
        base = got[0] if k < 3 else got[3]
        outs = []
        for flags in (0, _native.MW_FLAG_INDEX64):
            outs.append(torch.zeros_like(f.state))
            _native.call("mw_dirstage_f64", nx, nz, p["dx"], p["dz"], p["dt"], *bg, _native.ptr(f.src_w),
                         _native.ptr(base), _native.ptr(got[k]), _native.ptr(outs[-1]), p["dt"] / (3 - k % 3), d, 1, flags,
                         _native.stream_handle())
        assert torch.equal(outs[0], outs[1])
        assert max(normwise(got[k + 1].cpu().numpy(), outs[0].cpu().numpy())) <= TOL_STAGE, k


def test_steps_under_graph_capture():
    p = dict(make_params(100, 50, "thermal"), f64_mode="split")
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
