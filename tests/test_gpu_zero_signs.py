"""Solution variables of a cell with zero momentum: the quotient keeps the sign
of the zero, as a division does."""
import numpy as np
import pytest
import torch

from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.post import compute_solution_variables
from tests.helpers import make_params

pytestmark = pytest.mark.gpu


def test_quotients_of_zeros():
    p = make_params(64, 8, "collision")
    f = initialize_fields(p)
    init(f, p)
    rng = np.random.default_rng(3)
    zeros = torch.from_numpy(np.where(rng.random((2, 8, 64)) < 0.5, -0.0, 0.0)).cuda()
    f.state[1:3, 2:-2, 2:-2] = zeros
    f.state[0, 2:6, 2:-2] = -2.5 * f.hy_dens_cell[2:6, None]  # negative densities too
    got = compute_solution_variables(p, f).cpu().numpy()
    s = f.state.cpu().numpy()[:, 2:-2, 2:-2]
    ref = s[1:3] / (s[0] + f.hy_dens_cell.cpu().numpy()[2:-2, None])
    assert (got[1:3] == 0).all() and np.array_equal(np.signbit(got[1:3]), np.signbit(ref))
