"""Grids of short rows: solution variables over blocks of several rows, against
NumPy in extended precision, and in a time that follows the cells, not the rows."""
import numpy as np
import pytest
import torch

from pyminiweather_gb300.post import compute_solution_variables
from tests.test_gpu_diagnostics import developed, exact

pytestmark = pytest.mark.gpu


# rows per block: 256 of 2 to 8 columns, then 2048 / nx; rows that fill their last block and that do not
@pytest.mark.parametrize("nx,nz", [(2, 1), (2, 256), (3, 257), (7, 511), (8, 600), (31, 67), (64, 33), (683, 4), (1024, 3),
                                   (1025, 3), (2048, 2), (2049, 2)])
def test_solution_variables(nx, nz):
    p, f = developed(nx, nz)
    v = exact(p, f)[2]
    got = compute_solution_variables(p, f).cpu().numpy()
    for q in range(4):  # bounds of test_gpu_diagnostics.py
        scale = np.abs(v[q]).max() if q < 3 else 300.0
        assert np.abs(got[q] - v[q]).max() <= 4 * 2.0 ** -53 * scale, q


def us(fn):
    for _ in range(3):
        fn()
    times = []
    for _ in range(10):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            fn()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) / 5 * 1e3)
    return min(times)


def test_time_follows_the_cells():
    """16 columns take the time of 1024: the same cells, a row's constants per 16 cells more (12 operations beside
    16 x 12, 6 %) and rows that are not whole sectors; a factor of two is allowed."""
    short, long = developed(16, 64 * 1024), developed(1024, 1024)
    assert us(lambda: compute_solution_variables(*short)) <= 2.0 * us(lambda: compute_solution_variables(*long))
