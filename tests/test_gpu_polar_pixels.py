"""Polar grids on both sides of the rule that forms a tile in runs of columns or pixel by pixel, against the FP64 oracle:
fully sampled and coarse angle steps, tiles too wide for the fast path, long waves, squint, and a grid whose near
and far tiles differ.

Tolerance 1e-5: the split policy's bound.
"""
import numpy as np
import pytest

from conftest import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CASES = {
    # name: frequency, half the track (m), first range, dr, nr, u0, du, nu
    "sampled": (9.6e9, 50.0, 6000.0, 0.6, 70, -0.1, 5e-5, 100),
    "edge": (9.6e9, 50.0, 6000.0, 0.6, 70, -0.1, 1.8e-4, 100),
    "coarse": (9.6e9, 50.0, 6000.0, 0.6, 70, 0.3, 3e-4, 45),
    "wide": (9.6e9, 50.0, 6000.0, 0.8, 70, -0.05, 1e-3, 61),
    "long_wave": (4.35e8, 50.0, 6000.0, 0.8, 70, -0.1, 5e-4, 77),
    "near_and_far": (9.6e9, 30.0, 3100.0, 3.0, 400, -0.02, 2e-4, 50),
    "track_along_x": (9.6e9, -300.0, 6000.0, 0.6, 40, 0.2, 1e-3, 40),
}


@pytest.mark.parametrize("split", [1, 3])
@pytest.mark.parametrize("name", CASES)
def test_polar_tiles_match_the_fp64_oracle(name, split):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import build, core
    from oracle import reference as ora
    build.build()
    fc, half, r0, dr, nr, u0, du, nu = CASES[name]
    pulses, data_dr, k = 40, 0.8327, 4 * np.pi * fc / 299792458.0
    rng = np.random.default_rng(len(name))
    pos = rng.normal(0.0, 0.02, (pulses, 3)) + [0.0, 0.0, 3000.0]
    pos[:, 0 if half < 0 else 1] += np.linspace(-half, half, pulses)
    origin = (0.0, 0.0, 3000.0)
    start = r0 - abs(half) - 5.0
    samples = int((nr * dr + 2 * abs(half)) / data_dr) + 12
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    weight, phase = rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)
    ref = ora.bp_polar(data, pos, np.array(origin), r0, dr, nr, u0, du, nu, start, data_dr, k, weight, phase, 1, c128=True)[1]
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, weight, phase)]
    grid = core.Grid(origin, r0, dr, nr, u0, du, nu)
    images = [core.direct_polar(*args, grid, start, data_dr, k, pulse_split=split, chunk_pulses=c) for c in (64, 7)]
    assert torch.equal(*images)  # the image does not depend on the chunks
    assert rel_err(ref, images[0].cpu().numpy()) <= 1e-5
