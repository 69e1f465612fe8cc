"""FFBP leaves through both leaf kernels: two threads per run of columns (a program of a single leaf has few tiles) and one
(the batch kernel).  Both match the FP64 oracle and each other bit for bit: the same operations in the same order.
The cases are the edges of a run: partial last runs, window offsets (odd and even rows of the image), runs that
cross range bins, expansions that do not hold, windows that do not fit.

Tolerance 1e-5: the split policy's bound.
"""
from types import SimpleNamespace

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
    # name: pulses, nr, nu, dr, du, u0, data_dr, axis of the track, pulse spacing, k, wobble
    "short_leaf": (16, 130, 13, 0.25, 0.00416, -0.06, 0.8327, 1, 0.1, 402.0, 0.01),
    "long_leaf": (64, 33, 67, 0.25, 0.00099, 0.01, 0.8327, 1, 0.1, 402.0, 0.01),
    "one_pixel": (5, 1, 1, 0.25, 0.004, 0.1, 0.8327, 1, 0.1, 402.0, 0.01),
    "squint_along_x": (16, 40, 24, 0.3, 0.004, 0.6, 0.8327, 0, 0.1, 402.0, 0.01),
    "bins_aligned": (33, 64, 16, 0.5, 0.001, -0.3, 0.5, 1, 0.1, 402.0, 0.01),
    "coarse_angle": (3, 37, 11, 0.25, 0.03, -0.15, 0.8327, 0, 0.2, 402.0, 0.01),
    "undersampled": (40, 45, 30, 0.25, 0.006, -0.1, 0.8327, 1, 0.5, 402.0, 0.01),
    "wide_windows": (4, 128, 8, 2.0, 0.004, 0.0, 0.25, 1, 0.1, 402.0, 0.01),
    "steep_squint": (37, 70, 21, 0.25, 0.0168, 0.6, 0.8327, 1, 0.1, 402.0, 0.02),
    "long_wave": (21, 50, 27, 1.0, 0.0179, 0.35, 2.0, 1, 0.5, 18.2, 0.05),
    "mixed_runs": (18, 40, 30, 1.0, 0.0179, -0.1, 2.0, 1, 0.5, 18.2, 0.4),
}


@pytest.mark.parametrize("name", CASES)
def test_both_leaf_kernels_match_the_fp64_oracle(lib, name):
    from bp_project_gb300 import core
    from bp_project_gb300.batch import FFBPScene, SceneBatch
    from bp_project_gb300.gpu_backend import NodePlan
    from oracle import reference as ora
    pulses, nr, nu, dr, du, u0, data_dr, axis, step, k, wobble = CASES[name]
    rng = np.random.default_rng(len(name))
    pos = rng.normal(0.0, wobble, (pulses, 3)) + [5.0, -3.0, 3000.0]
    pos[:, axis] += step * (np.arange(pulses) - 0.5 * pulses)
    origin, r0 = pos.mean(axis=0), 4000.3
    start = r0 - 0.5 * pulses * step - 3.0 * data_dr  # the first bins' taps leave the row for some pixels
    samples = int((nr * dr + pulses * step) / data_dr) + 12
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    weight, phase = rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)
    ref = ora.bp_polar(data, pos, origin, r0, dr, nr, u0, du, nu, start, data_dr, k, weight, phase, 1, c128=True)[1]
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, weight, phase)]
    node = NodePlan(0, 0, pulses, origin, r0, dr, nr, u0, du, nu, 1)
    for cr, cu in (((0, nr), (0, nu)), ((nr // 3, nr), (nu // 2, nu))):
        two = core.FFBPProgram([node], cr, cu).execute(*args, start, data_dr, k)
        assert rel_err(ref[cr[0]:cr[1], cu[0]:cu[1]], two.cpu().numpy()) <= 1e-5
        plan = SimpleNamespace(nodes=lambda: [node], shape=(cr[1] - cr[0], cu[1] - cu[0]), crop_r=cr, crop_u=cu)
        batch = SceneBatch([FFBPScene(*args, start, data_dr, k, plan=plan)])
        batch.execute()
        assert torch.equal(batch.outputs[0], two)
        batch.close()
