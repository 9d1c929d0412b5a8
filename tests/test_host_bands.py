"""How many row bands the host-buffer step takes (no GPU needed)."""
import pytest

from pyminiweather_gb300 import _native


@pytest.mark.parametrize("nx,nz,nbands,bands", [
    (8192, 4096, 32, 32), (8192, 4096, 100, 64), (8192, 4096, 1, 1), (8192, 4096, 0, 1), (2048, 1024, 32, 4),
    (2050, 1031, 32, 4), (4100, 1300, 3, 3),
    (1024, 1024, 32, 2), (1024, 1023, 32, 1),  # a band has 2^19 cells or more
    (70000, 40, 32, 2), (2000000, 31, 32, 1),  # and 16 rows or more
    (100, 50, 32, 1)])
def test_bands(nx, nz, nbands, bands):
    L = _native.load()
    for mode in (_native.MW_F64_IEEE, _native.MW_F64_SPLIT):
        assert L.mw_host_step_bands(nx, nz, mode, nbands) == bands
    assert L.mw_host_step_bands(nx, nz, _native.MW_F64_NATIVE, nbands) == 1


def test_bad_arguments():
    L = _native.load()
    assert L.mw_host_step_bands(1, 64, _native.MW_F64_IEEE, 8) == 0
    assert L.mw_host_step_bands(64, 64, 9, 8) == 0
