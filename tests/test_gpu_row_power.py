"""The row constants' power (rho theta)^gamma of the IEEE x stage, by the pressure
it gives: every entry of its logarithm's and exponential's tables, the ends of
its range and the arguments beyond, against 50-digit arithmetic."""
from decimal import Decimal, getcontext

import numpy as np
import pytest
import torch

from pyminiweather_gb300 import _native
from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from tests.helpers import make_params

pytestmark = pytest.mark.gpu

C0, GAMMA = Decimal(27.5629410929725921310572974482), Decimal(1.40027894002789400278940027894)
NX = 8
SHAPE = np.array([0.05, -0.04, 0.09, -0.08, 0.02, 0.1, -0.1, -0.03])  # (rho theta)' over its background along a row


def arguments():
    """A value in every 64th of an octave and at its ends, over octaves that meet every 64th of the power's."""
    x = []
    for j in range(64):
        for k, t in enumerate((0.0, 0.37, 0.999)):
            x.append((1.0 + (j + t) / 64) * 2.0 ** ((7 * j + 3 * k) % 29 - 14))
    x += [20.0, 300.0, 400.0, 1.0, np.nextafter(1.0, 0), np.nextafter(2.0, 0)]
    # the ends of the range that the tables take, and beyond
    return x + [1.3 * 2.0 ** e for e in (-660, -651, -650, -649, -300, 300, 648, 649, 650, 651, 660)]


def test_pressure_of_rows_vs_exact():
    getcontext().prec = 50
    rt = np.array(arguments())
    nz = len(rt)
    p = make_params(NX, nz, "thermal")
    f = initialize_fields(p)
    init(f, p)
    f.hy_dens_cell.fill_(1.0)
    f.hy_dens_theta_cell.fill_(1.0)
    f.hy_dens_theta_cell[2:-2] = torch.from_numpy(rt).to(f.device)
    f.state.zero_()
    pert = rt[:, None] * SHAPE[None, :]
    f.state[3, 2:-2, 2:-2] = torch.from_numpy(pert).to(f.device)
    out = torch.zeros_like(f.state)
    _native.call("mw_dirstage_f64", NX, nz, p["dx"], p["dz"], p["dt"], *[_native.ptr(a) for a in f.backgrounds()], None,
                 _native.ptr(f.state), _native.ptr(f.state), _native.ptr(out), p["dt"], 0, _native.MW_F64_IEEE, 0,
                 _native.stream_handle())
    got = out[1, 2:-2, 2:-2].cpu().numpy()
    c = Decimal(p["dt"]) / Decimal(p["dx"])
    for k in range(nz):
        bg, s = Decimal(float(rt[k])), [Decimal(float(v)) for v in pert[k]]
        flux = []
        for i in range(NX):  # interface i between cells i - 1 and i of the periodic row
            a = (7 * (s[i - 1] + s[i]) - (s[i - 2] + s[(i + 1) % NX])) / 12
            flux.append(C0 * ((bg + a) ** GAMMA - bg ** GAMMA))
        scale = max(abs(v) for v in flux)
        for i in range(NX):
            exact = c * (flux[i] - flux[(i + 1) % NX])
            # a flux: the power 1, its factors 4, the interpolated value 3 roundings of 16 / 12 of the largest, twice
            # (series and slope) and the series 4: below 20; the difference of two, one more
            assert abs(Decimal(float(got[k, i])) - exact) <= 42 * Decimal(2.0 ** -53) * c * scale, (k, rt[k], i)


@pytest.mark.parametrize("rt", (1e-30, 1e-60, 1e40))
def test_totals_over_extreme_backgrounds(rt):
    """Internal energy Cv (C0 / p0)^(Rd / Cp) (rho theta)^gamma of a row whose coefficients leave the normal range."""
    from pyminiweather_gb300.post import compute_stats
    getcontext().prec = 50
    p = make_params(NX, 3, "thermal")
    f = initialize_fields(p)
    init(f, p)
    f.hy_dens_cell.fill_(1.0)
    f.hy_dens_theta_cell.fill_(rt)
    f.state.zero_()
    f.state[3, 2:-2, 2:-2] = torch.from_numpy(rt * SHAPE).to(f.device)
    k = Decimal(717.0) * (Decimal("27.5629410929725921310572974482") / Decimal(1e5)) ** (Decimal(287.0) / Decimal(1004.0))
    vals = [Decimal(rt) + Decimal(float(v)) for v in rt * SHAPE]
    exact = 3 * sum(k * v ** GAMMA for v in vals) * Decimal(p["dx"]) * Decimal(p["dz"])
    # a term: (C0 / p0)^(Rd / Cp) and the power 2 each, products, series and sums below 20
    assert abs(Decimal(compute_stats(p, f)[1]) - exact) <= 30 * Decimal(2.0 ** -53) * exact
