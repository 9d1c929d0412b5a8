"""The IEEE form carries fluxes over the hyperviscosity coefficient: the rounded
numbers that scale them there and back must not make every flux too large or too
small.  The mass flux of a stage, with the hyperviscosity and all else zero, over
many grids: its factor against dt / d in extended precision, from so many cells
that their own roundings average out."""
import numpy as np
import pytest
import torch

from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from tests.helpers import make_params

pytestmark = pytest.mark.gpu

N = 256  # cells each way; the errors of 65536 values of about an ulp each: 0.004 ulp of their mean factor


def factor_error(f, p, spacing, dt, direction):
    """Relative error of the mass flux's factor dt / spacing in one stage of momenta that are integers."""
    q = dict(p, dx=spacing, dz=spacing)
    out, zero = torch.empty_like(f.state), torch.zeros_like(f.state)
    _native.call("mw_dirstage_f64", N, N, q["dx"], q["dz"], q["dt"], *[_native.ptr(a) for a in f.backgrounds()], None,
                 _native.ptr(zero), _native.ptr(f.state), _native.ptr(out), dt, direction, _native.MW_F64_IEEE, 0,
                 _native.stream_handle())
    s = f.state[1 + direction].cpu().numpy().astype(np.int64)
    s = s[2:-2, 2:-2] if direction == 0 else s[2:-2, 2:-2].T
    a = 7 * (s[:, 1:-2] + s[:, 2:-1]) - s[:, :-3] - s[:, 3:]  # 12 x the value at the interfaces inside the row
    want = (a[:, :-1] - a[:, 1:]).astype(np.longdouble) * (np.longdouble(dt) / (12 * np.longdouble(spacing)))
    got = out[0].cpu().numpy()
    got = got[2:-2, 2:-2] if direction == 0 else got[2:-2, 2:-2].T
    diff = got[:, 2:-2].astype(np.longdouble) - want
    return float((diff * want).sum() / (want * want).sum())


@pytest.mark.parametrize("direction", (0, 1))
def test_mass_flux_keeps_its_factor(direction):
    p = make_params(N, N, "thermal")
    f = initialize_fields(p)
    init(f, p)
    f.state.zero_()
    gen = torch.Generator(device=f.device).manual_seed(1)
    f.state[1 + direction, 2:-2, 2:-2] = torch.randint(-2 ** 20, 2 ** 20, (N, N), generator=gen, device=f.device,
                                                       dtype=torch.float64)
    errors = []
    for n in range(41, 6000, 149):
        d = 2e4 / n
        p["dt"] = d * 1.5 / 450.0
        for div in (3, 2, 1):
            errors.append(factor_error(f, p, d, p["dt"] / div, direction))
    e = np.abs(errors) * 2.0 ** 53
    print("factor errors x 2^53: mean %.3f largest %.3f of %d" % (e.mean(), e.max(), len(e)))
    # dt / (12 d) formed by two rounded operations has up to 2 and 0.5 on average
    assert e.max() <= 1.2 and e.mean() <= 0.35
