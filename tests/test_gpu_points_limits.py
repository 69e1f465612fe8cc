"""Split-precision direct BP at points whose tiles lie at the limits of the fast path, against the FP64 oracle.

Tolerance 1e-5: the split policy's bound.
"""
import numpy as np
import pytest

from conftest import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import build
    build.build()


def raster(rows, cols, step, x0):
    i, j = np.divmod(np.arange(rows * cols), cols)
    return np.column_stack([x0 + step * i, step * (j - 0.5 * cols), 0.1 * np.sin(1.0 * j)])


def error(xyz, altitude, spacing, dr, k, pulses=40):
    from bp_project_gb300 import core
    from oracle import reference as ora
    rng = np.random.default_rng(len(xyz))
    pos = np.column_stack([np.zeros(pulses), spacing * (np.arange(pulses) - 0.5 * pulses), np.full(pulses, altitude)])
    r = np.linalg.norm(xyz[None] - pos[::pulses - 1, None], axis=2)
    start = float(r.min()) - 20.0 * dr
    samples = int((r.max() - start) / dr) + 20
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    w, ph = rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)
    _, ref = ora.backproject_points(data, pos, xyz, start, dr, k, w, ph, c128=True)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, w, ph, xyz)]
    return rel_err(ref, core.backproject_points(*args, start, dr, k).cpu().numpy())


@pytest.mark.parametrize("step", [120.0, 132.0, 160.0])
def test_offsets_beyond_the_integer_range(lib, step):
    """A tile of 500 points in a line, up to 30, 33 and 40 km from its centre, seen from 10,000 km at a wavelength of
    63 m: the fast path's offsets are 32-bit integers of 2^-16 m, which end at 32.8 km."""
    assert error(raster(1, 500, step, 3.0e6), 1.0e7, 1000.0, 200.0, 0.2) <= 1e-5


@pytest.mark.parametrize("rows,cols,step", [(60, 60, 0.5), (40, 300, 0.1), (22, 23, 1.0)])
def test_short_range(lib, rows, cols, step):
    """400 MHz from 40 m height and 40 to 80 m ground range: the range series' third order is up to 1e-3 rad there."""
    assert error(raster(rows, cols, step, 40.0), 40.0, 0.1, 0.5, 4 * np.pi * 4e8 / 299792458.0) <= 1e-5


def test_wide_tiles_at_a_long_wavelength(lib):
    """Tiles of 33 km half-width from 360 km, k = 1e-5: the same order is 3e-3 bins of 400 m."""
    assert error(raster(60, 60, 2000.0, 3.0e5), 2.0e5, 100.0, 400.0, 1e-5) <= 1e-5


@pytest.mark.parametrize("altitude,x0,step,cols,dr", [(223.0, 200.0, 0.1, 300, 0.2), (3000.0, 3.0e4, 0.5, 120, 0.4164),
                                                      (3000.0, 3.0e4, 0.25, 300, 0.4164)])
def test_rasters_at_near_and_far_ranges(lib, altitude, x0, step, cols, dr):
    """9.6 GHz at 300 m, where tiles may have a radius of 6 m, and at 30 km, where 61 m fit: taken in spatial order or not."""
    assert error(raster(20, cols, step, x0), altitude, 0.05, dr, 402.0) <= 1e-5


@pytest.mark.parametrize("altitude,x0,gap", [(223.0, 200.0, 5.0), (3000.0, 3.0e4, 20.0), (3000.0, 3.0e4, 80.0)])
def test_patches_at_near_and_far_ranges(lib, altitude, x0, gap):
    """Patches of 170 points `gap` apart, three to a tile: formed whole where the tile fits, patch by patch where it does not."""
    n = np.arange(1000)
    rng = np.random.default_rng(7)
    xyz = np.column_stack([x0 + gap * (n // 170) + rng.uniform(-0.5, 0.5, 1000), rng.uniform(-0.5, 0.5, 1000), 0.0 * n])
    assert error(xyz, altitude, 0.05, 0.4, 402.0) <= 1e-5
