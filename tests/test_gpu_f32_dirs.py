"""The FP32 direction kernels take a direction's three RK stages in one launch:
rows and columns at the edges of tiles, runs and warps, rows of any alignment,
against the oracle's FP64 time steps, halos and state_tmp included."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ensemble import Ensemble, member_params
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.solve import evolve, reset_direction
from tests.helpers import BACKGROUNDS, make_params, normwise

pytestmark = pytest.mark.gpu

# A stage rounds the state (2^-25 of max|s|) and adds dt / dx = 1/300 of flux differences whose largest part, the
# pressure perturbation of a 20 K bubble (1e4 Pa), carries about four FP32 roundings against momenta of ~5:
# 1e4 x 4 x 6e-8 / 300 / 5 = 1.6e-6 of max|s| a stage, 3e-5 over the 18 stages of three steps.
TOL = 3e-5
GRIDS = [(2, 1), (3, 2), (5, 1), (11, 7), (12, 8), (13, 9), (116, 16), (117, 17), (127, 23), (128, 33), (129, 40),
         (244, 50), (245, 64), (257, 100), (488, 31), (489, 37), (1001, 130), (64, 515), (130, 1030)]


def developed(p, seed):
    f = initialize_fields(p, dtype=torch.float32)
    init(f, p)
    rng = np.random.default_rng(seed)
    noise = rng.standard_normal(f.shape) * np.array([1e-3, 5.0, 2.0, 0.5])[:, None, None]
    f.state += torch.from_numpy(noise).to(f.device, torch.float32)
    f.state_tmp.copy_(f.state + 0.5)
    return f


def oracle_of(p, f, reverse):
    o = O.OracleSim(O.make_params(p["nx"], p["nz"], p["ic_type"]))
    for name in BACKGROUNDS:
        getattr(o, name)[:] = getattr(f, name).cpu().numpy()
    o.state[:], o.state_tmp[:] = f.state.double().cpu().numpy(), f.state_tmp.double().cpu().numpy()
    o.reverse = int(reverse)
    if f.src_w is not None:
        o.src_w[:] = f.src_w.cpu().numpy()
    return o


@pytest.mark.parametrize("nx,nz", GRIDS)
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


@pytest.mark.parametrize("nx,nz", [(2, 1), (37, 13), (250, 125), (1030, 300)])
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


@pytest.mark.parametrize("z_tile", (1, 5, 16, 64))
def test_ensemble_members_vs_oracle(z_tile):
    sizes = [(2, 1), (64, 32), (65, 66), (245, 130), (37, 13)]
    ens = Ensemble([(member_params(nx, nz), None) for nx, nz in sizes], dtype=torch.float32, z_tile=z_tile)
    sims = []
    for e, (nx, nz) in enumerate(sizes):
        p = make_params(nx, nz, "thermal")
        f = developed(p, e)
        ens.member_state(e).copy_(f.state)
        ens.member_state_tmp(e).copy_(f.state_tmp)
        sims.append(oracle_of(p, f, False))
    ens.step(1)
    ens.step(2)
    for e, o in enumerate(sims):
        o.evolve(3)
        assert max(normwise(ens.member_state(e).double().cpu().numpy(), o.state, interior=False)) <= TOL, e
        assert max(normwise(ens.member_state_tmp(e).double().cpu().numpy(), o.state_tmp, interior=False)) <= TOL, e


def by_stages(p, f, nsteps):
    """Time steps issued stage by stage (mw_dirstage_f32), z then x first; returns state and state_tmp."""
    s, t, a = f.state.clone(), f.state_tmp.clone(), torch.zeros_like(f.state)
    bg = [_native.ptr(b) for b in f.backgrounds()]
    for n in range(nsteps):
        for d in (1, 0) if n % 2 == 0 else (0, 1):
            for frc, out, div in ((s, a, 3), (a, t, 2), (t, s, 1)):
                _native.call("mw_dirstage_f32", f.nx, f.nz, p["dx"], p["dz"], p["dt"], *bg, _native.ptr(f.src_w),
                             _native.ptr(s), _native.ptr(frc), _native.ptr(out), p["dt"] / div, d, 1,
                             _native.stream_handle())
    return s, t


@pytest.mark.parametrize("nx,nz,same", [(66, 600000, False), (43_000_001, 1, True)])
def test_long_columns_and_rows_vs_stages(nx, nz, same):
    """A column of many tiles; a row too long for the direction kernels, which is stepped stage by stage."""
    if torch.cuda.mem_get_info()[0] < 12 * 4 * (nx + 4) * (nz + 4) * 4:
        pytest.skip("not enough device memory")
    p = dict(make_params(nx, nz, "thermal", xlen=20.0 * nx, zlen=1e4 if nz > 1 else 20.0))
    f = initialize_fields(p, dtype=torch.float32)
    init(f, p)
    g = torch.Generator(device="cuda").manual_seed(3)
    for q, amp in enumerate((1e-3, 5.0, 2.0, 0.5)):
        f.state[q] += amp * torch.randn(f.shape[1:], device="cuda", generator=g)
    ref, ref_tmp = by_stages(p, f, 2)
    reset_direction()
    evolve(p, f, None, dt=p["dt"], nsteps=2)
    for got, want in ((f.state, ref), (f.state_tmp, ref_tmp)):
        got, want = got[:, 2:-2, 2:-2], want[:, 2:-2, 2:-2]
        if same:
            assert torch.equal(got, want)
        else:
            for q in range(4):
                assert (got[q] - want[q]).abs().max() <= TOL * want[q].abs().max(), q
