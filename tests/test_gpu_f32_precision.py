"""The FP32 form's steps take a direction's three RK stages in one launch: they
are no further from FP64 than the same steps issued stage by stage."""
import pytest
import torch

from pyminiweather_gb300.data import initialize_fields
from pyminiweather_gb300.ics import init
from pyminiweather_gb300.solve import evolve, reset_direction
from tests.helpers import make_params, rel_l2
from tests.test_gpu_f32_dirs import by_stages

pytestmark = pytest.mark.gpu


# Line kernels (the first two grids) and direction kernels, each over enough steps that the errors are those of the
# arithmetic and not of chance: the two sides' rounding errors are sums over at least 20000 cells and 600 stages,
# so their norms repeat to a few per cent; 5 % is allowed.
@pytest.mark.parametrize("ic,nx,nz,nsteps", [("density-current", 200, 100, 200), ("collision", 512, 256, 100),
                                             ("collision", 1024, 512, 200)])
def test_no_further_from_fp64_than_the_stage_kernels(ic, nx, nz, nsteps):
    p = make_params(nx, nz, ic)
    f = initialize_fields(p, dtype=torch.float32)
    init(f, p)
    exact = initialize_fields(dict(p, f64_mode="native"))
    init(exact, p)
    exact.state.copy_(f.state)
    stages, _ = by_stages(p, f, nsteps)
    reset_direction()
    evolve(p, f, None, dt=p["dt"], nsteps=nsteps)
    reset_direction()
    evolve(dict(p, f64_mode="native"), exact, None, dt=p["dt"], nsteps=nsteps)
    reset_direction()
    ref = exact.state.cpu().numpy()
    err, bar = rel_l2(f.state.cpu().numpy(), ref), rel_l2(stages.cpu().numpy(), ref)
    for q in range(4):
        assert err[q] <= 1.05 * bar[q], (q, err, bar)
