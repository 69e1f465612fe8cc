"""A polar image onto ground lattices of odd sizes and steps, against the FP64 oracle's evaluation.

Tolerance 1e-5: the split policy's bound.  The offsets from a tile's centre are two-float; places in the image are
FP32 over at most 60 bins (4e-6 bins against an image of independent values, whose slope is about 2 per bin).
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import build
    build.build()


@pytest.mark.parametrize("rows,cols,step_row,step_col", [
    (1, 1, (0.5, 0.0, 0.0), (0.0, 0.5, 0.0)), (33, 37, (0.5, 0.0, 0.0), (0.0, 0.5, 0.0)),
    (65, 31, (0.31, 0.1, 0.0), (-0.07, 0.43, 0.0)), (40, 70, (-0.3, 0.2, 0.0), (0.2, 0.3, 0.0)),
    (50, 20, (0.0, 0.6, 0.0), (0.1, 0.0, 0.0))])
def test_lattice_evaluation_matches_the_fp64_oracle(lib, rows, cols, step_row, step_col):
    from bp_project_gb300 import core
    from oracle import reference as ora
    rng = np.random.default_rng(rows)
    origin, r0, dr, u0, du, k = (5.0, -3.0, 3000.0), 4000.3, 0.5, -0.02, 2e-4, 402.0
    nr, nu = 180, 260
    img = (rng.standard_normal((nr, nu)) + 1j * rng.standard_normal((nr, nu))).astype(np.complex64)
    lat0 = (5.0 + np.sqrt((r0 + 45.0) ** 2 - 3000.0 ** 2), 2.0, 0.0)
    pts = (np.array(lat0) + np.arange(rows)[:, None, None] * np.array(step_row) +
           np.arange(cols)[None, :, None] * np.array(step_col)).reshape(-1, 3)
    ref = np.asarray(ora.evaluate_image(img, origin, r0, dr, u0, du, pts, k, c128=True)[1]).reshape(rows, cols)
    assert np.linalg.norm(ref) > 0.0
    grid = core.Grid(origin, r0, dr, nr, u0, du, nu, 1)
    out = core.evaluate_lattice(torch.from_numpy(img).cuda(), grid, lat0, step_row, step_col, rows, cols, k).cpu().numpy()
    assert np.linalg.norm(out - ref) <= 1e-5 * np.linalg.norm(ref)
