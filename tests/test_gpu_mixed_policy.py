"""The mixed policy's FP64 steps (root, bin and phase reduction of their own) where they can go wrong, against the
FP64 oracle: rows of 3, 4 and 5 samples (no, one and two supported bins), a row of more bins than the fast
bin's integer field, points that run off both ends of the row, points at an image's origin and outside it.

Tolerance 1e-6 (the mixed policy rounds weights, sine, cosine and sums to FP32: a few 6e-8 each); what the
oracle has no support for is exactly zero.
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


@pytest.mark.parametrize("samples,dr", [(3, 4.0), (4, 4.0), (5, 4.0), (200, 0.5), (600000, 0.01)])
def test_points_across_the_row(lib, samples, dr):
    from bp_project_gb300 import core
    from oracle import reference as ora
    rng = np.random.default_rng(samples)
    start, k = 1000.0, 402.0
    pos = np.column_stack([np.zeros(9), np.linspace(-2, 2, 9), np.full(9, 700.0)])
    end = start + dr * samples
    r = np.concatenate([rng.uniform(start - 2 * dr, end + 2 * dr, 500), rng.uniform(start, start + 3 * dr, 100),
                        rng.uniform(end - 4 * dr, end, 100)])
    xyz = np.column_stack([np.sqrt(r**2 - 699.0**2), rng.uniform(-3, 3, r.size), rng.uniform(0, 1, r.size)])
    data = (rng.standard_normal((9, samples)) + 1j * rng.standard_normal((9, samples))).astype(np.complex64)
    weight, phase = rng.uniform(0.5, 1.5, 9), rng.uniform(-9, 9, 9)
    _, ref = ora.backproject_points(data, pos, xyz, start, dr, k, weight, phase, c128=True)
    out = core.backproject_points(*[torch.from_numpy(a).cuda() for a in (data, pos, weight, phase, xyz)], start, dr, k,
                                  mode="mixed").cpu().numpy()
    zero = np.abs(ref) == 0
    assert zero.any() and np.all(out[zero] == 0)
    if samples == 3:
        assert zero.all()
    else:
        assert rel_err(ref, out) <= 1e-6


def test_image_at_its_origin_and_outside(lib):
    from bp_project_gb300 import core
    from oracle import reference as ora
    rng = np.random.default_rng(5)
    grid = core.Grid((10.0, -20.0, 600.0), 601.0, 0.5, 240, -0.9, 0.01, 180)
    image = (rng.standard_normal((240, 180)) + 1j * rng.standard_normal((240, 180))).astype(np.complex64)
    xyz = np.column_stack([rng.uniform(10.0, 450.0, 3000), rng.uniform(-400.0, 400.0, 3000), np.zeros(3000)])
    xyz[:3] = [10.0, -20.0, 0.0]  # the origin's ground point
    ref = np.asarray(ora.evaluate_image(image, grid.origin, grid.r0, grid.dr, grid.u0, grid.du, xyz, 402.0))
    out = core.evaluate_image(torch.from_numpy(image).cuda(), grid, torch.from_numpy(xyz).cuda(), 402.0).cpu().numpy()
    zero = np.abs(ref) == 0
    assert zero[:3].all() and (~zero).any() and np.all(out[zero] == 0)
    assert rel_err(ref, out) <= 1e-6
