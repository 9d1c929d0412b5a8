"""The FP32 line kernels take a direction's three RK stages in one launch (grids
whose rows and columns fit a CTA): lengths at the edges of warps, runs and
pieces against the oracle's time steps, halos and state_tmp included, and, bit
for bit, against the direction kernels, which ensembles always take; the
direction kernels themselves on ragged grids above the line kernels' limit.

Tolerance: the direction kernels' (test_gpu_f32_dirs.py), the arithmetic being
theirs: 1.6e-6 of max|s| a stage, 3e-5 over the 18 stages of three steps."""
import pytest
import torch

from pyminiweather_gb300.ensemble import Ensemble, member_params
from pyminiweather_gb300.solve import evolve, reset_direction
from tests.helpers import make_params, normwise
from tests.test_gpu_f32_dirs import TOL, developed, oracle_of

pytestmark = pytest.mark.gpu

LINES = [(2, 1), (3, 2), (4, 3), (31, 30), (32, 31), (33, 32), (62, 63), (63, 62), (64, 64), (100, 50), (481, 37),
         (37, 481), (993, 20), (20, 993), (24, 2000), (2000, 24), (5, 9000), (9000, 5), (401, 199), (600, 500)]
DIRS = [(1001, 301), (2501, 131), (130, 2400), (244, 1240), (489, 640)]


@pytest.mark.parametrize("nx,nz", LINES + DIRS)
@pytest.mark.parametrize("ic,reverse", [("collision", False), ("gravity", True)])
def test_steps_vs_oracle(ic, reverse, nx, nz):
    p = make_params(nx, nz, ic)
    f = developed(p, nx * 1000 + nz)
    o = oracle_of(p, f, reverse)
    reset_direction(reverse)
    evolve(p, f, None, dt=p["dt"], nsteps=1)
    evolve(p, f, None, dt=p["dt"], nsteps=2)
    reset_direction()
    o.evolve(3)
    assert max(normwise(f.state.double().cpu().numpy(), o.state, interior=False)) <= TOL
    assert max(normwise(f.state_tmp.double().cpu().numpy(), o.state_tmp, interior=False)) <= TOL


@pytest.mark.parametrize("nx,nz", [(2, 1), (31, 30), (100, 50), (245, 130), (401, 199), (512, 256)])
def test_bits_of_the_direction_kernels(nx, nz):
    ens = Ensemble([(member_params(nx, nz), None)], dtype=torch.float32)
    p = make_params(nx, nz, "thermal")
    f = developed(p, 7)
    ens.member_state(0).copy_(f.state)
    ens.member_state_tmp(0).copy_(f.state_tmp)
    reset_direction()
    evolve(p, f, None, dt=p["dt"], nsteps=3)
    reset_direction()
    ens.step(3)
    assert torch.equal(ens.member_state(0), f.state) and torch.equal(ens.member_state_tmp(0), f.state_tmp)


def test_steps_under_graph_capture():
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
