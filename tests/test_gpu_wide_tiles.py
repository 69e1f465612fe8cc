"""Lattices whose tiles are too wide for the fast path (every pulse in two-float), against the FP64 oracle: steps from 1.5 m up
at 4 km, rows in either direction, tilted, more pulses than a chunk, both halves of a block.

Tolerance 1e-5: the split policy's bound.
"""
import numpy as np
import pytest

from conftest import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pulses", [1, 2, 67])
@pytest.mark.parametrize("step_row,step_col", [((1.5, 0, 0), (0, 1.5, 0)), ((-7.0, 0.3, 0), (0.2, 5.0, 0)),
                                               ((2.0, 0, 0.7), (0.1, 2.0, -0.4))])
def test_wide_lattice_tiles(step_row, step_col, pulses):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import build, core
    from oracle import reference as ora
    build.build()
    rng = np.random.default_rng(pulses)
    rows, cols, dr, k = 45, 37, 0.8328, 402.0
    pos = np.column_stack([np.zeros(pulses), 0.1 * (np.arange(pulses) - 0.5 * pulses), np.full(pulses, 3000.0)])
    origin, sr, sc = np.array([2900.0, -40.0, 0.0]), np.array(step_row), np.array(step_col)
    pts = (origin + np.arange(rows)[:, None, None] * sr + np.arange(cols)[None, :, None] * sc).reshape(-1, 3)
    r = np.linalg.norm(pts[None] - pos[:, None], axis=2)
    start = float(r.min()) - 3.0 * dr  # the first bins' taps leave the row for part of the image
    samples = int((r.max() - r.min()) / dr) + 5
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    weight, phase = rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)
    _, ref = ora.backproject_points(data, pos, pts, start, dr, k, weight, phase, c128=True)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, weight, phase)]
    img = core.backproject_lattice(*args, tuple(origin), tuple(sr), tuple(sc), rows, cols, start, dr, k, pulse_split=1)
    assert rel_err(ref, img.cpu().numpy().ravel()) <= 1e-5
