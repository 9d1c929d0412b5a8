"""The IEEE-FP64 line kernels on the smallest grids: a warp's two halves take
two variables each of sixteen slots, fourteen cells a run.  Lengths at the
edges of those runs against the oracle's time steps, halos and state_tmp
included.

Tolerance: the arithmetic of a value is that of the whole slots; as there
(test_gpu_fp64_lines.py), 18 stages of at most 3e-14 of max|s|: 6e-13."""
import pytest
import torch

from oracle import oracle as O
from pyminiweather_gb300.solve import evolve, reset_direction
from tests.helpers import BACKGROUNDS, make_params, normwise
from tests.test_gpu_fp64_lines import TOL, developed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(2, 3), (13, 14), (14, 13), (15, 16), (16, 15), (27, 29), (28, 28), (29, 27), (42, 43),
                                   (43, 57), (57, 42), (75, 70), (120, 40), (100, 50)])
@pytest.mark.parametrize("ic,reverse", [("collision", False), ("gravity", True)])
def test_steps_vs_oracle(ic, reverse, nx, nz):
    p = make_params(nx, nz, ic)
    f = developed(p, nx * 1000 + nz)
    o = O.OracleSim(O.make_params(nx, nz, ic))
    for name in BACKGROUNDS:
        getattr(o, name)[:] = getattr(f, name).cpu().numpy()
    o.state[:], o.state_tmp[:], o.reverse = f.state.cpu().numpy(), f.state_tmp.cpu().numpy(), int(reverse)
    if f.src_w is not None:
        o.src_w[:] = f.src_w.cpu().numpy()
    reset_direction(reverse)
    evolve(p, f, None, dt=p["dt"], nsteps=1)
    evolve(p, f, None, dt=p["dt"], nsteps=2)
    reset_direction()
    o.evolve(3)
    assert max(normwise(f.state.cpu().numpy(), o.state, interior=False)) <= TOL
    assert max(normwise(f.state_tmp.cpu().numpy(), o.state_tmp, interior=False)) <= TOL


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nonfinite_reaches_the_cells_of_the_stage_kernels(bad):
    """A NaN or Inf spreads to the cells that the reference's formulas reach (the native form's), in a step."""
    got = []
    for mode in ("fp64", "native"):
        p = dict(make_params(60, 30, "thermal"), f64_mode=mode)
        f = developed(p, 1)
        f.state[2, 17, 31] = bad
        reset_direction()
        evolve(p, f, None, dt=p["dt"], nsteps=1)
        got.append(torch.isfinite(f.state[:, 2:-2, 2:-2]).cpu())
    reset_direction()
    assert torch.equal(got[0], got[1])
