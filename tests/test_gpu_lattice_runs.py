"""Split-precision lattice tiles (runs of eight rows per thread, the block's halves on alternate
pulses) where the run expansion and the halves can go wrong, against the FP64 oracle.

Tolerance 1e-5: the split policy's bound.  The run's fifth-order remainder and the folded fourth-order
term stay below 0.004 / (K R) rad inside the precision envelope (2e-7 rad at K R = 2e4, the
nearest case here), and the FP32 sums add about 1e-6.
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


@pytest.mark.parametrize("pulses", [1, 2, 3, 65])
@pytest.mark.parametrize("geometry", ["rows_cross", "rows_along", "rows_back", "tilted", "near"])
def test_lattice_runs_match_the_fp64_oracle(lib, geometry, pulses):
    from bp_project_gb300 import core
    from oracle import reference as ora
    rng = np.random.default_rng(pulses)
    near, dr, k = (300.0, 0.5, 402.0) if geometry == "near" else (4000.0, 0.8328, 402.0)
    pos = np.zeros((pulses, 3))
    pos[:, 1] = 0.1 * (np.arange(pulses) - 0.5 * pulses)
    pos[:, 2] = 0.75 * near
    x0 = np.sqrt(near**2 - pos[0, 2]**2) + 20.0
    step = {"rows_cross": ((0.5, 0, 0), (0, 0.5, 0)), "rows_along": ((0, 0.6, 0), (0.4, 0.1, 0)),
            "rows_back": ((-0.5, 0.02, 0), (0.03, -0.5, 0)), "tilted": ((0.5, 0, 0.11), (0, 0.5, -0.07)),
            "near": ((0.1, 0, 0), (0, 0.1, 0))}[geometry]
    rows, cols = 45, 37
    sr, sc = (np.array(v) for v in step)
    origin = np.array([x0 + 40.0, -12.0, 0.0])
    pts = (origin + np.arange(rows)[:, None, None] * sr + np.arange(cols)[None, :, None] * sc).reshape(-1, 3)
    r = np.linalg.norm(pts[None] - pos[:, None], axis=2)
    start = float(r.min()) - 3.0 * dr  # the first bins' taps leave the row for part of the image
    samples = int((r.max() - r.min()) / dr) + 5
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    weight, phase = rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)
    _, ref = ora.backproject_points(data, pos, pts, start, dr, k, weight, phase, c128=True)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, weight, phase)]
    for split in sorted({1, min(2, pulses)}):
        img = core.backproject_lattice(*args, tuple(origin), tuple(sr), tuple(sc), rows, cols, start, dr, k,
                                       pulse_split=split)
        err = rel_err(ref, img.cpu().numpy().ravel())
        assert err <= 1e-5, (geometry, pulses, split, err)
