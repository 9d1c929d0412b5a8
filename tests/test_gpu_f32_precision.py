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


@pytest.mark.parametrize("nx,nz", [(100, 50), (401, 199), (1001, 301)])  # line kernels (2), direction kernels
@pytest.mark.parametrize("ic", ["collision", "gravity"])
def test_one_rounding_of_the_state_a_direction(ic, nx, nz):
    """rho w in [64, 128) and a step so short that the increments' own errors (F ~ 1e4 Pa, dt / dz = 3e-6, four
    roundings of 2^-24: 8e-9) are a thousandth of the state's ulp, 2^-17: what is left is the rounding of the state at
    the end of either direction, half an ulp each, whatever gravity and the forcing of w add."""
    p = make_params(nx, nz, ic)
    f = initialize_fields(p, dtype=torch.float32)
    init(f, p)
    g = torch.Generator(device="cuda").manual_seed(nx)
    f.state[0].normal_(0.0, 1e-2, generator=g)
    f.state[2].uniform_(80.0, 112.0, generator=g)
    exact = initialize_fields(dict(p, f64_mode="native"))
    init(exact, p)
    exact.state.copy_(f.state)
    if ic == "gravity":
        f.src_w.normal_(0.0, 0.1, generator=g)
        exact.src_w.copy_(f.src_w)
    reset_direction()
    evolve(p, f, None, dt=1e-3 * p["dt"])
    reset_direction()
    evolve(dict(p, f64_mode="native"), exact, None, dt=1e-3 * p["dt"])
    reset_direction()
    got, ref = f.state[2, 2:-2, 2:-2].double(), exact.state[2, 2:-2, 2:-2]
    assert ref.min() >= 64 and ref.max() < 128
    assert (got - ref).abs().max() <= 1.02 * 2.0 ** -17
