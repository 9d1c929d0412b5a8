"""Totals and solution variables at the edges of their kernels' row pieces and
blocks, against NumPy in extended precision, with non-finite and extreme
values passed through as a division would."""
import numpy as np
import pytest
import torch

from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.post import compute_solution_variables, compute_stats
from tests.helpers import make_params

pytestmark = pytest.mark.gpu

CP, CV, RD, P0 = 1004.0, 717.0, 287.0, 1.0e5
C0, GAMMA = 27.5629410929725921310572974482, 1.40027894002789400278940027894


def developed(nx, nz, dtype=torch.float64):
    p = make_params(nx, nz, "collision")
    f = initialize_fields(p, dtype=dtype)
    init(f, p)
    rng = np.random.default_rng(nx * 7 + nz)
    noise = rng.standard_normal(f.shape) * np.array([1e-3, 5.0, 2.0, 0.5])[:, None, None]
    f.state += torch.from_numpy(noise).to(f.device, dtype)
    return p, f


def exact(p, f):
    ld = np.longdouble
    s = f.state.double().cpu().numpy().astype(ld)[:, 2:-2, 2:-2]
    hr = f.hy_dens_cell.cpu().numpy().astype(ld)[2:-2, None]
    hrt = f.hy_dens_theta_cell.cpu().numpy().astype(ld)[2:-2, None]
    rho = s[0] + hr
    th = (s[3] + hrt) / rho
    e = (s[1] ** 2 + s[2] ** 2) / rho + rho * CV * th / (P0 / (C0 * (rho * th) ** ld(GAMMA))) ** (ld(RD) / CP)
    area = ld(p["dx"]) * p["dz"]
    return rho.sum() * area, e.sum() * area, np.stack([s[0], s[1] / rho, s[2] / rho, th - hrt / hr])


@pytest.mark.parametrize("nx,nz", [(2, 1), (31, 3), (32, 16), (33, 17), (100, 50), (257, 1025), (2047, 33), (2049, 20),
                                   (4100, 2100)])
def test_totals_and_variables(nx, nz):
    p, f = developed(nx, nz)
    m, e, v = exact(p, f)
    gm, ge = compute_stats(p, f)
    # positive sums of N terms, each good to ~10 roundings, added in trees and runs of at most ~N / 2^18 terms
    tol = 2.0 ** -53 * (10 + nx * nz / 2.0 ** 18)
    assert abs(gm - m) <= tol * m and abs(ge - e) <= tol * e
    got = compute_solution_variables(p, f).cpu().numpy()
    # roundings: u, w two (rho, the quotient); theta', as the reference forms it, is the difference of two thetas
    # near 300 of one and three roundings
    for q in range(4):
        scale = np.abs(v[q]).max() if q < 3 else 300.0
        assert np.abs(got[q] - v[q]).max() <= 4 * 2.0 ** -53 * scale, q


def test_fp32_totals():
    p, f = developed(130, 70, torch.float32)
    m, e, _ = exact(p, f)
    gm, ge = compute_stats(p, f)
    assert abs(gm - m) <= 1e-14 * m and abs(ge - e) <= 1e-14 * e


def test_quotients_of_extreme_values():
    p, f = developed(64, 8)
    rng = np.random.default_rng(1)
    f.state[1, 2:-2, 2:-2] = torch.from_numpy(rng.standard_normal((8, 64)) * 10.0 ** rng.uniform(-320, 308, (8, 64)))
    f.state[2, 2, 2:8] = torch.tensor([float("inf"), float("-inf"), float("nan"), 0.0, -0.0, 5e-324])
    f.state[0, 3, 5] = -f.hy_dens_cell[3]  # rho = 0
    f.state[0, 4, 5] = float("inf")
    got = compute_solution_variables(p, f).cpu().numpy()
    s = f.state.cpu().numpy()[:, 2:-2, 2:-2]
    with np.errstate(all="ignore"):
        rho = s[0] + f.hy_dens_cell.cpu().numpy()[2:-2, None]
        for q in (1, 2):
            ref = s[q] / rho
            assert np.array_equal(np.isnan(got[q]), np.isnan(ref))
            ok = ~np.isnan(ref)
            fin = ok & np.isfinite(ref)
            assert np.array_equal(got[q][ok & ~fin], ref[ok & ~fin])
            assert (np.abs(got[q][fin] - ref[fin]) <= np.spacing(np.abs(ref[fin]))).all()
