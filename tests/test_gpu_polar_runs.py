"""Direct BP on polar grids in runs of eight angle columns (two half blocks on alternate pulses) where the run
expansion, the shared window entry and the fallbacks can go wrong, against the FP64 oracle.

Tolerance 1e-5: the split policy's bound.  The expansion drops at most 1e-7 turns (6e-7 rad), the slope of
the phase along a run is FP32 (below 1e-7 of at most half a turn per column here: 3e-7 turns at a run's end),
and the FP32 sums add about 1e-6.
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


CASES = {
    # name: pulses, nr, nu, r0, dr, du, u0, data_dr, axis of the track, pulse spacing, side
    "root_grid": (200, 70, 83, 4000.3, 0.25, 6e-5, -0.02, 0.8327, 1, 0.5, 1),
    "one_pixel": (3, 1, 1, 4000.3, 0.25, 6e-5, 0.1, 0.8327, 1, 0.1, 1),
    "along_x_left": (65, 40, 37, 4000.3, 0.3, 1e-4, 0.5, 0.8327, 0, 0.5, -1),
    "tall_tiles": (33, 131, 9, 4000.3, 0.25, 0.0019, 0.0, 0.8327, 1, 0.1, 1),
    "bins_aligned": (64, 64, 16, 4000.0, 0.5, 2e-4, -0.3, 0.5, 1, 0.5, 1),
    "undersampled": (64, 33, 40, 4000.3, 0.25, 5e-4, 0.1, 0.8327, 1, 0.5, 1),   # runs cross bins
    "near": (17, 34, 21, 300.0, 0.05, 4e-4, 0.05, 0.2, 1, 0.05, 1),
    "outside_envelope": (9, 130, 40, 400.0, 1.0, 0.0019, 0.0, 0.8327, 1, 0.5, 1),  # two-float fallback
}


@pytest.mark.parametrize("name", CASES)
def test_polar_runs_match_the_fp64_oracle(lib, name):
    from bp_project_gb300 import core
    from oracle import reference as ora
    pulses, nr, nu, r0, dr, du, u0, data_dr, axis, step, side = CASES[name]
    rng = np.random.default_rng(len(name))
    pos = rng.normal(0.0, 0.01, (pulses, 3)) + [5.0, -3.0, 0.7 * r0]
    pos[:, axis] += step * (np.arange(pulses) - 0.5 * pulses)
    origin, k = pos.mean(axis=0), 402.0
    start = r0 - 0.5 * pulses * step - 3.0 * data_dr  # the first bins' taps leave the row for some pixels
    samples = int((nr * dr + pulses * step) / data_dr) + 12
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    weight, phase = rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)
    ref = ora.bp_polar(data, pos, origin, r0, dr, nr, u0, du, nu, start, data_dr, k, weight, phase, side, c128=True)[1]
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, weight, phase)]
    grid = core.Grid(tuple(origin), r0, dr, nr, u0, du, nu, side)
    images = [core.direct_polar(*args, grid, start, data_dr, k, chunk_pulses=c).cpu().numpy() for c in (64, 7)]
    assert np.array_equal(*images)  # the image does not depend on the chunks
    images.append(core.direct_polar(*args, grid, start, data_dr, k, pulse_split=min(2, pulses)).cpu().numpy())
    for img in images[1:]:
        err = rel_err(ref, img)
        assert err <= 1e-5, (name, err)
