"""The IEEE-FP64 x pass cuts a row into runs of blocks of 64 cells and takes
what a block's first cell needs from the block before: rows whose length lies
at the edges of blocks and runs, against the oracle's direction-stage.  The
result must not depend on how the rows are cut (the cut depends on the number
of rows), bit for bit."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from tests.helpers import BACKGROUNDS, make_params, normwise

pytestmark = pytest.mark.gpu

# One stage adds to a state of order max|s| increments dt / dx (F(i) - F(i+1)), dt / dx = 1/300, whose terms carry
# a few dozen roundings of 2^-53 of their largest part (the pressure perturbation, at most ~2e4 Pa against momenta
# of ~10): below 40 x 2^-53 x 2e4 / 10 / 300 = 3e-14 of max|s|; the repository's bar for one stage is 1e-12.
TOL_STAGE = 1e-12
NXS = (2, 3, 5, 61, 62, 63, 64, 65, 125, 126, 127, 128, 190, 191, 1021, 1022, 1023, 1025, 2047)


def developed(p, seed):
    f = initialize_fields(p)
    init(f, p)
    rng = np.random.default_rng(seed)
    noise = rng.standard_normal(f.shape) * np.array([1e-3, 5.0, 2.0, 0.5])[:, None, None]
    f.state += torch.from_numpy(noise).to(f.device)
    return f


def stage(p, f, state, direction, flags):
    frc, out = state.clone(), torch.zeros_like(state)
    _native.call("mw_dirstage_f64", f.nx, f.nz, p["dx"], p["dz"], p["dt"], *[_native.ptr(a) for a in f.backgrounds()],
                 _native.ptr(f.src_w), _native.ptr(state), _native.ptr(frc), _native.ptr(out), p["dt"] / 2, direction,
                 _native.MW_F64_IEEE, flags, _native.stream_handle())
    return frc, out


@pytest.mark.parametrize("nx", NXS)
@pytest.mark.parametrize("ic,nz", [("collision", 7), ("gravity", 33)])
def test_stage_at_block_edges_vs_oracle(ic, nz, nx):
    p = make_params(nx, nz, ic)
    f = developed(p, nx)
    o = O.OracleSim(O.make_params(nx, nz, ic))
    for name in BACKGROUNDS:  # the same backgrounds on both sides, to the last bit
        getattr(o, name)[:] = getattr(f, name).cpu().numpy()
    for direction in (0, 1):
        frc, out = stage(p, f, f.state, direction, 1)
        ofrc, oout = f.state.cpu().numpy().copy(), np.zeros(f.shape)
        o.dirstage(f.state.cpu().numpy(), ofrc, oout, p["dt"] / 2, direction)
        assert max(normwise(out.cpu().numpy(), oout)) <= TOL_STAGE, (direction, nx)
        assert np.array_equal(frc.cpu().numpy(), ofrc)  # halo writes


@pytest.mark.parametrize("nx", (100, 401, 1500, 3001))
def test_rows_do_not_depend_on_the_cut(nx):
    """An x stage of many rows and of each few of them give the same bits."""
    nz = 640
    p = make_params(nx, nz, "collision")
    f = developed(p, nx)
    _, whole = stage(p, f, f.state, 0, 0)
    for r0, n in ((0, 1), (5, 3), (100, 40)):
        q = dict(make_params(nx, n, "collision"), dx=p["dx"], dz=p["dz"], dt=p["dt"])
        g = initialize_fields(q)
        g.hy_dens_cell.copy_(f.hy_dens_cell[r0:r0 + n + 4])
        g.hy_dens_theta_cell.copy_(f.hy_dens_theta_cell[r0:r0 + n + 4])
        for a in (g.hy_dens_int, g.hy_dens_theta_int, g.hy_pressure_int):
            a.fill_(1.0)  # not read by the x pass
        part = f.state[:, r0:r0 + n + 4].contiguous()
        _, out = stage(q, g, part, 0, 0)
        assert torch.equal(out[:, 2:-2, 2:-2], whole[:, r0 + 2:r0 + n + 2, 2:-2]), (r0, n)


@pytest.mark.parametrize("mode", ("fp64", "split"))
@pytest.mark.parametrize("nx,nz,nbands", [(2050, 1031, 32), (4100, 1300, 3)])
def test_host_step_bands_of_ragged_grids(nx, nz, nbands, mode):
    """Grids large enough for several bands, whose rows do not divide by them: evolve_host gives the bits of
    copy in, evolve, copy out, in both direction orders."""
    import pyminiweather_gb300.solve.step as S
    p = dict(make_params(nx, nz, "collision"), f64_mode=mode)
    a, b = developed(p, 3), developed(p, 3)
    h = b.state.cpu().pin_memory()
    for step in range(2):
        S.reverse_direction = bool(step)
        S.evolve(p, a, None, dt=p["dt"])
        S.reverse_direction = bool(step)
        S.evolve_host(p, b, h, h, dt=p["dt"], nbands=nbands)
        torch.cuda.synchronize()
        assert torch.equal(h, a.state.cpu()) and torch.equal(a.state_tmp, b.state_tmp), step
    S.reset_direction()
