"""The z stage adjoint in one kernel: tiles of 32 columns by 1 to 29 rows
(the rule takes 5 rows on the small grids here, 13 to 29 on the wide ones),
against the two-kernel adjoint of the reference's formulas, at the edges of
the tiles, with a wall inside, at the edge of and next to a tile.

Tolerance: an adjoint is a chain of at most 40 rounded FP64 operations whose
terms exceed the sum at most 8 times (7 + 1 of the interpolation, 3 + 1 of
the third difference): 40 x 8 x 2^-53 = 3.6e-14 of the largest value, either
side; 1e-13 covers both."""
import pytest
import torch

from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.solve import evolve
from tests.helpers import make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(32, 5), (33, 6), (31, 1), (65, 11), (2000, 25), (2400, 41), (1000, 116),
                                   (1025, 117)])
def test_stage_vjp_z_tiles(nx, nz):
    p = make_params(nx, nz, "collision")
    f = initialize_fields(p)
    init(f, p, None)
    evolve(dict(p, f64_mode="native"), f, None, dt=p["dt"], nsteps=2)
    s = f.state.clone()
    gen = torch.Generator(device="cpu").manual_seed(nx * 1000 + nz)
    g = torch.zeros_like(s)
    g[:, 2:-2, 2:-2] = torch.randn(4, nz, nx, generator=gen, dtype=torch.float64).to(s.device)
    ws = torch.empty(int(_native.load().mw_dirstage_vjp_workspace_bytes(nx, nz)) // 8 + 1, dtype=torch.float64,
                     device=s.device)
    hb = [_native.ptr(a) for a in f.backgrounds()]
    outs = []
    for mode in (0, 2):
        out = torch.full_like(s, 7.0)
        _native.call("mw_dirstage_vjp_f64", nx, nz, p["dx"], p["dz"], p["dt"], *hb, _native.ptr(s), _native.ptr(g),
                     None, None, 0, _native.ptr(out), p["dt"] / 2, 1, mode, _native.ptr(ws), ws.numel() * 8,
                     _native.stream_handle())
        outs.append(out)
    ref, got = outs
    for v in range(4):
        err = float((got[v] - ref[v]).abs().max() / ref[v].abs().max().clamp_min(1e-300))
        assert err <= 1e-13, (nx, nz, v, err)
    frame = torch.ones_like(got, dtype=torch.bool)
    frame[:, 2:-2, 2:-2] = False
    assert float(got[frame].abs().max()) == 0.0
