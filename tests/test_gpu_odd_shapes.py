"""Grids of a few columns, a few rows or many more of one than of the other: the
kernels' other shapes of work, and that a call's time follows its cells.

Times are the least of ten, compared within one process with those of another
grid; a bound lies between the ratio measured and the one before, both beside it."""
import numpy as np
import pytest
import torch

from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.post import compute_solution_variables
from pyminiweather_gb300.solve import evolve
from pyminiweather_gb300.solve import step as step_module
from tests import test_gpu_diagnostics as diagnostics
from tests.helpers import make_params
from tests.test_gpu_short_rows import us

pytestmark = pytest.mark.gpu


def developed(nx, nz):
    p = make_params(nx, nz, "collision")
    f = initialize_fields(p)
    init(f, p)
    gen = torch.Generator(device=f.device).manual_seed(nx * 7 + nz)
    noise = torch.randn(f.shape, generator=gen, device=f.device, dtype=torch.float64)
    f.state += noise * torch.tensor([1e-3, 5.0, 2.0, 0.5], device=f.device, dtype=torch.float64)[:, None, None]
    return p, f


class Vjp:
    """The adjoint of one stage at a developed state."""

    def __init__(self, nx, nz):
        self.p, self.f = developed(nx, nz)
        self.g = torch.zeros_like(self.f.state)
        gen = torch.Generator(device=self.g.device).manual_seed(nx * 1000 + nz)
        self.g[:, 2:-2, 2:-2] = torch.randn(4, nz, nx, generator=gen, dtype=torch.float64, device=self.g.device)
        n = int(_native.load().mw_dirstage_vjp_workspace_bytes(nx, nz))
        self.ws = torch.empty(n // 8 + 1, dtype=torch.float64, device=self.g.device)
        self.out = torch.empty_like(self.g)

    def __call__(self, mode, direction):
        p, f = self.p, self.f
        _native.call("mw_dirstage_vjp_f64", f.nx, f.nz, p["dx"], p["dz"], p["dt"],
                     *[_native.ptr(a) for a in f.backgrounds()], _native.ptr(f.state), _native.ptr(self.g), None, None,
                     0, _native.ptr(self.out), p["dt"] / 2, direction, _native.F64_MODES[mode], _native.ptr(self.ws),
                     self.ws.numel() * 8, _native.stream_handle())
        return self.out


def frame_max(a):
    a = a.clone()
    a[:, 2:-2, 2:-2] = 0.0
    return float(a.abs().max())


@pytest.mark.parametrize("mode", ("split", "fp64"))
@pytest.mark.parametrize("nx,nz", [(2, 1), (2, 300), (3, 2), (300, 2), (4097, 1), (70001, 3), (130, 70)])
def test_adjoint_clears_the_halo(nx, nz, mode):
    v = Vjp(nx, nz)
    for direction in (0, 1):
        v.out.fill_(7.0)
        assert frame_max(v(mode, direction)) == 0.0, direction


def test_adjoint_of_long_rows_takes_the_time_of_its_cells():
    long, square = Vjp(3000000, 2), Vjp(3000, 2000)  # 398 us against 377; a CTA to a halo row 1640
    assert us(lambda: long("split", 0)) <= 2.0 * us(lambda: square("split", 0))


# widths and rows of a tile: 2 to 32 columns of narrow grids, 64 and 128 of flat ones; whole, cut and single-row tiles,
# stretches with an interface less and without any
@pytest.mark.parametrize("nx,nz", [(2, 1), (2, 3), (2, 509), (2, 510), (2, 4000), (3, 1100), (5, 70), (7, 253), (8, 125),
                                   (9, 126), (15, 1000), (16, 61), (17, 62), (40, 700), (66, 900), (100, 500), (255, 200),
                                   (4000, 1), (5000, 2), (3001, 5), (70000, 6), (3000, 7), (3000, 8)])
def test_adjoint_z_tiles(nx, nz):
    """Against the adjoint of the reference's formulas, to the bound derived in test_gpu_adjoint_tiles.py."""
    v = Vjp(nx, nz)
    ref, got = v("native", 1).clone(), v("fp64", 1)
    for q in range(4):
        err = float((got[q] - ref[q]).abs().max() / ref[q].abs().max().clamp_min(1e-300))
        assert err <= 1e-13, (q, err)
    assert frame_max(got) == 0.0


def test_adjoint_of_few_columns_takes_the_time_of_its_cells():
    narrow, square = Vjp(2, 100000), Vjp(500, 400)  # 78 us against 60; in tiles of 32 columns 594
    assert us(lambda: narrow("fp64", 1)) <= 3.0 * us(lambda: square("fp64", 1))


def stage(p, f, mode, direction=0):
    out = torch.zeros_like(f.state)
    _native.call("mw_dirstage_f64", f.nx, f.nz, p["dx"], p["dz"], p["dt"], *[_native.ptr(a) for a in f.backgrounds()],
                 None, _native.ptr(f.state), _native.ptr(f.state), _native.ptr(out), p["dt"] / 2, direction,
                 _native.F64_MODES[mode], 0, _native.stream_handle())
    return out


# runs that end in the first and in the second half of a block, of one to nine blocks; one to four runs a warp, whose
# rows end within and with a CTA; rows that are cut into as many runs as there can be
@pytest.mark.parametrize("nx,nz", [(2, 1), (2, 9), (2, 40001), (5, 20003), (29, 9731), (30, 9730), (31, 9729), (62, 40),
                                   (66, 9000), (94, 5000), (95, 5001), (200, 3000), (257, 2000), (478, 1300), (510, 700),
                                   (511, 700), (542, 700), (4000, 16), (20000, 2)])
def test_x_stage(nx, nz):
    """The IEEE x stage against the reference's formulas.  A stage adds to a state increments whose terms are sums of
    at most a few dozen rounded operations on values up to (7 + 7 + 1 + 1) / 12 of the state's or the pressure's range
    (test_gpu_fp64_runs.py, which states the bar of 1e-12 for one stage)."""
    p, f = developed(nx, nz)
    ref, got = stage(p, f, "native"), stage(p, f, "fp64")
    for q in range(4):
        a, b = got[q, 2:-2, 2:-2], ref[q, 2:-2, 2:-2]
        assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max()), q


def test_x_stage_of_short_rows_takes_the_time_of_its_slots():
    # rows of 30 + 2 slots of 32 that a warp's instruction takes, against 62 + 2: 675 us against 1404, in blocks of 64
    # slots always 1246
    short, full = developed(30, 200000), developed(62, 200000)
    assert us(lambda: stage(*short, "fp64")) <= 0.7 * us(lambda: stage(*full, "fp64"))


# pieces of a row of 256 cells and more, up to 2048, whole and cut
@pytest.mark.parametrize("nx,nz", [(255, 2), (257, 2), (512, 300), (513, 303), (4000, 16), (20000, 2), (40961, 9),
                                   (300000, 1), (700001, 1)])
def test_solution_variables_of_long_rows(nx, nz):
    p, f = diagnostics.developed(nx, nz)
    v = diagnostics.exact(p, f)[2]
    got = compute_solution_variables(p, f).cpu().numpy()
    for q in range(4):  # bounds of test_gpu_diagnostics.py
        scale = np.abs(v[q]).max() if q < 3 else 300.0
        assert np.abs(got[q] - v[q]).max() <= 4 * 2.0 ** -53 * scale, q


@pytest.mark.parametrize("mode", ("fp64", "split"))
@pytest.mark.parametrize("nx,nz", [(4096, 20), (4097, 20), (20, 4097), (5000, 13), (13, 5000), (100, 5000)])
def test_recorded_step_of_long_lines(nx, nz, mode):
    """A recorded step gives the bits of a step, and its last stage of a direction is the direction's result."""
    p, f = developed(nx, nz)
    q = dict(p, f64_mode=mode, step_flags=0)
    stages, out = torch.zeros((6,) + tuple(f.shape), dtype=torch.float64, device=f.device), torch.zeros_like(f.state)
    for reverse in (0, 1):
        s0 = f.state.clone()
        _native.call("mw_step_record_f64", nx, nz, p["dx"], p["dz"], p["dt"], p["dt"],
                     *[_native.ptr(a) for a in f.backgrounds()], None, _native.ptr(s0), _native.ptr(stages),
                     _native.ptr(out), reverse, _native.F64_MODES[mode], _native.stream_handle())
        step_module.reverse_direction = bool(reverse)
        evolve(q, f, None, dt=p["dt"])
        step_module.reset_direction()
        inner = (slice(None), slice(2, -2), slice(2, -2))
        assert torch.equal(stages[0][inner], s0[inner])
        if mode == "fp64":  # the first stage of a double-FP32 step stays a pair where it is not recorded
            assert torch.equal(out[inner], f.state[inner])
        else:
            scale = f.state[inner].abs().amax(dim=(1, 2))
            assert bool(((out[inner] - f.state[inner]).abs().amax(dim=(1, 2)) <= 1e-12 * scale).all())
