"""FFBP leaf tiles (runs of eight angle columns per thread) where the run expansion, the shared window
entry and the fallbacks can go wrong: a program of a single leaf against the FP64 oracle.

Tolerance 1e-5: the split policy's bound.  The expansion drops at most 5e-8 turns (3e-7 rad), the
place in the window is within 1e-6 bins (offsets up to 8 bins in FP32), and the FP32 sums add about 1e-6.
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
    # name: pulses, nr, nu, dr, du, u0, data_dr, axis of the track, pulse spacing
    "short_leaf": (16, 130, 13, 0.25, 0.00416, -0.06, 0.8327, 1, 0.1),
    "long_leaf": (64, 33, 67, 0.25, 0.00099, 0.01, 0.8327, 1, 0.1),
    "one_pixel": (5, 1, 1, 0.25, 0.004, 0.1, 0.8327, 1, 0.1),
    "squint_along_x": (16, 40, 24, 0.3, 0.004, 0.6, 0.8327, 0, 0.1),
    "bins_aligned": (33, 64, 16, 0.5, 0.001, -0.3, 0.5, 1, 0.1),
    "coarse_angle": (3, 37, 11, 0.25, 0.03, -0.15, 0.8327, 0, 0.2),      # the expansion does not hold
    "undersampled": (40, 45, 30, 0.25, 0.006, -0.1, 0.8327, 1, 0.5),    # a run spans several bins
    "wide_windows": (4, 128, 8, 2.0, 0.004, 0.0, 0.25, 1, 0.1),         # a pulse's window does not fit
}


@pytest.mark.parametrize("name", CASES)
def test_leaf_runs_match_the_fp64_oracle(lib, name):
    from bp_project_gb300 import core
    from bp_project_gb300.gpu_backend import NodePlan
    from oracle import reference as ora
    pulses, nr, nu, dr, du, u0, data_dr, axis, step = CASES[name]
    rng = np.random.default_rng(len(name))
    pos = rng.normal(0.0, 0.01, (pulses, 3)) + [5.0, -3.0, 3000.0]
    pos[:, axis] += step * (np.arange(pulses) - 0.5 * pulses)
    origin, r0, k = pos.mean(axis=0), 4000.3, 402.0
    start = r0 - 0.5 * pulses * step - 3.0 * data_dr  # the first bins' taps leave the row for some pixels
    samples = int((nr * dr + pulses * step) / data_dr) + 12
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    weight, phase = rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)
    ref = ora.bp_polar(data, pos, origin, r0, dr, nr, u0, du, nu, start, data_dr, k, weight, phase, 1, c128=True)[1]
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, weight, phase)]
    node = NodePlan(0, 0, pulses, origin, r0, dr, nr, u0, du, nu, 1)
    for cr, cu in (((0, nr), (0, nu)), ((nr // 3, nr), (nu // 2, nu))):  # whole, and a window at odd offsets
        img = core.FFBPProgram([node], cr, cu).execute(*args, start, data_dr, k)
        err = rel_err(ref[cr[0]:cr[1], cu[0]:cu[1]], img.cpu().numpy())
        assert err <= 1e-5, (name, cr, cu, err)
