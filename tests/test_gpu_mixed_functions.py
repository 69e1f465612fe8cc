"""The mixed policy's own root and phase reduction over their range, against extended precision: one pulse, data of ones,
so that a point's value is exp(i (k d + phase)).

Tolerance 1e-6 at phases of up to 1e9 rad: there the roundings of d, of k in quarter turns and of their product are 1.1e-7
rad each (2^-53 of 1e9), the interpolation weights, sine and cosine in FP32 a few 6e-8.  A root a few last bits off, or
a reduction to the wrong quarter, would show.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def cuda(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, np.float64))).cuda()


# 1e-18 to 1e18 m: the squares run through the FP32 exponents and off both ends (the library's root).
@pytest.mark.parametrize("scale", [1e-18, 1e-6, 1.0, 4e3, 1e6, 1e12, 1e18])
@pytest.mark.parametrize("turns", [0.0, 1.0, 1e3, 1e9])
def test_root_and_phase(scale, turns):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import build, core
    build.build()
    rng = np.random.default_rng(3)
    xyz = rng.standard_normal((4000, 3))
    xyz *= (scale * rng.uniform(1.0, 1.9, 4000) / np.linalg.norm(xyz, axis=1))[:, None]
    phase = rng.uniform(-3.0, 3.0)
    k = turns / scale
    data = torch.ones((1, 4), dtype=torch.complex64, device="cuda")  # one supported bin: scale <= d < 2 scale
    out = core.backproject_points(data, cuda([[0, 0, 0]]), cuda([1]), cuda([phase]), cuda(xyz), 0.0, scale, k, mode="mixed")
    d = np.sqrt((xyz.astype(np.longdouble) ** 2).sum(axis=1))
    ang = np.longdouble(k) * d + np.longdouble(phase)
    want = np.cos(ang).astype(np.float64) + 1j * np.sin(ang).astype(np.float64)
    inside = (d >= scale * (1 + 1e-12)) & (d < 2 * scale * (1 - 1e-12))
    assert inside.sum() > 3900
    assert np.abs(out.cpu().numpy() - want)[inside].max() <= 1e-6


@pytest.mark.parametrize("scale", [1e-3, 1.0, 4e3, 1e9])
def test_image_coordinates(scale):
    """An image that is linear in range and angle gives a point's own coordinates: root and quotient, to the
    FP32 of the value (64 rows and columns; tolerance 1e-5 of 64)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import build, core
    build.build()
    rng = np.random.default_rng(4)
    n = 64
    grid = core.Grid((0.0, 0.0, 0.4 * scale), scale, scale / n, n, -0.9, 1.8 / n, n)
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    image = torch.from_numpy((i + 1j * j).astype(np.complex64)).cuda()
    r, u = scale * rng.uniform(1.1, 1.8, 4000), rng.uniform(-0.8, 0.8, 4000)
    g = np.sqrt(r**2 - (0.4 * scale) ** 2)
    xyz = np.column_stack([g * np.sqrt(1 - u**2), g * u, np.zeros(4000)])
    out = core.evaluate_image(image, grid, cuda(xyz), 0.0).cpu().numpy()
    assert np.abs(out - ((r - scale) * n / scale + 1j * (u + 0.9) * n / 1.8)).max() <= 1e-5 * n
