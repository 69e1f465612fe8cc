"""The mixed policy at the ends of a stencil's support: a point whose place is exactly bin 1 or bin n - 2 by division,
with steps whose product with the reciprocal rounds to the other side.  Bins 1 <= place < n - 2 have a value (ffbp.py:24-30),
as in the FP64 policy; everything else is exactly zero.

Tolerance 1e-6: the mixed policy's (weights, sine and cosine in FP32).
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


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, np.float64))).cuda()


@pytest.mark.parametrize("step,n", [(49.0, 8), (0.7, 9), (3.3, 9), (4.9, 7), (0.25, 8)])
def test_points_on_the_first_and_last_bins(lib, step, n):
    from bp_project_gb300 import core
    places = np.arange(n) * step
    want = (places / step >= 1) & (places / step < n - 2)
    xyz = np.column_stack([places, np.zeros(n), np.zeros(n)])
    data = torch.ones((1, n), dtype=torch.complex64, device="cuda")
    for mode in ("fp64", "mixed"):
        out = core.backproject_points(data, cuda([[0, 0, 0]]), cuda([1]), cuda([0]), cuda(xyz), 0.0, step, 0.0, mode=mode)
        out = out.cpu().numpy()
        assert np.array_equal(out != 0, want) and np.abs(out[want] - 1).max() <= 1e-6, mode


@pytest.mark.parametrize("step,n", [(49.0, 8), (0.7, 9), (3.3, 9), (4.9, 7)])
def test_images_on_the_first_and_last_rows(lib, step, n):
    from bp_project_gb300 import core
    grid = core.Grid((0.0, 0.0, 0.0), 0.0, step, n, -0.5, 0.125, 9)
    places = np.arange(1, n) * step
    want = (places / step >= 1) & (places / step < n - 2)
    image = torch.ones((n, 9), dtype=torch.complex64, device="cuda")
    out = core.evaluate_image(image, grid, cuda(np.column_stack([places, np.zeros(n - 1), np.zeros(n - 1)])), 0.0)
    out = out.cpu().numpy()
    assert np.array_equal(out != 0, want) and np.abs(out[want] - 1).max() <= 1e-6
