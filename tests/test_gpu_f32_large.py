"""The FP32 direction kernels on grids that take no line kernels (more than
300000 cells, or lines too long for them): rows at the edges of runs and warps
with eight and with four cells a lane, columns at the edges of tiles, against
the oracle's FP64 time steps, halos and state_tmp included."""
import pytest

from pyminiweather_gb300.solve import evolve, reset_direction
from tests.helpers import make_params, normwise
from tests.test_gpu_f32_dirs import TOL, developed, oracle_of

pytestmark = pytest.mark.gpu

# a run holds 244 cells with eight a lane, 116 with four (at most nine rows of 16000 and more)
GRIDS = [(244, 1231), (245, 1230), (487, 620), (488, 617), (489, 614), (732, 411), (733, 410), (1001, 301), (4097, 75),
         (16100, 9), (16125, 8), (20000, 2), (20001, 1), (127, 2400), (128, 2350), (129, 2330), (9, 33400), (300, 1021),
         (640, 513)]


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
