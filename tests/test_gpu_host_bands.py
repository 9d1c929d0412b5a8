"""The host-buffer step in several row bands (grids of more than 2^20 cells, by
the count the library gives): the bits of copy in, evolve, copy out for even and
ragged bands, both direction orders, page-locked and pageable arrays, in and out
of the same array, halo writes on and off; the finite check."""
import pytest
import torch

import pyminiweather_gb300.solve.step as S
from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from tests.helpers import make_params

pytestmark = pytest.mark.gpu


def bands(p, nbands):
    return _native.load().mw_host_step_bands(p["nx"], p["nz"], _native.F64_MODES[p["f64_mode"]], nbands)


def developed(p):
    f = initialize_fields(p)
    init(f, p)
    gen = torch.Generator(device=f.device).manual_seed(p["nx"])
    noise = torch.randn(f.shape, generator=gen, device=f.device, dtype=torch.float64)  # halo cells too
    f.state += noise * torch.tensor([1e-3, 5.0, 2.0, 0.5], device=f.device, dtype=torch.float64)[:, None, None]
    return f


@pytest.mark.parametrize("mode", ("fp64", "split"))
@pytest.mark.parametrize("nx,nz,nbands,want,flags,pinned,ic", [
    (1024, 1024, 2, 2, 1, True, "collision"), (1025, 1029, 8, 2, 0, True, "gravity"),
    (2050, 1031, 3, 3, 0, False, "collision"), (2048, 1024, 4, 4, 1, False, "gravity"),
    (70001, 40, 8, 2, 1, True, "collision"), (520, 8209, 8, 8, 0, True, "collision"),
    (3001, 1751, 10, 10, 1, True, "gravity"),  # from ten bands on the end ones are half as tall
    (3000, 2111, 64, 12, 0, False, "collision"), (600, 55931, 64, 64, 1, True, "collision")])
def test_bands_match_copy_step_copy(nx, nz, nbands, want, flags, pinned, ic, mode):
    p = dict(make_params(nx, nz, ic), f64_mode=mode, step_flags=flags)
    assert bands(p, nbands) == want
    a = developed(p)
    b = initialize_fields(p)
    init(b, p)
    h_in = a.state.cpu()
    h_in = h_in.pin_memory() if pinned else h_in
    h_out = torch.full_like(h_in, 7.0, pin_memory=pinned)
    a.state_tmp.copy_(b.state_tmp)
    for step in range(3):  # both direction orders; the later steps in and out of the same array
        S.reverse_direction = bool(step % 2)
        a.state.copy_(h_in if step == 0 else h_out)
        S.evolve(p, a, None, dt=p["dt"])
        S.reverse_direction = bool(step % 2)
        S.evolve_host(p, b, h_in if step == 0 else h_out, h_out, dt=p["dt"], nbands=nbands)
        torch.cuda.synchronize()
        assert torch.equal(h_out, a.state.cpu()), step
        assert torch.equal(a.state, b.state) and torch.equal(a.state_tmp, b.state_tmp), step
    S.reset_direction()


@pytest.mark.parametrize("mode", ("fp64", "split"))
def test_finite_check_with_bands(mode):
    p = dict(make_params(2050, 1031, "collision"), f64_mode=mode, check_finite=True)
    assert bands(p, 3) == 3
    f = initialize_fields(p)
    init(f, p)
    h = f.state.cpu().pin_memory()
    S.reset_direction()
    S.evolve_host(p, f, h, h, dt=p["dt"], nbands=3)
    torch.cuda.synchronize()
    h[2, 2 + 700, 2 + 11] = float("nan")
    with pytest.raises(_native.MiniWeatherError) as ei:
        S.evolve_host(p, f, h, h, dt=p["dt"], nbands=3)
    assert ei.value.status == 7
    torch.cuda.synchronize()
    S.reset_direction()
