"""The trajectory-update kernels against the same steps as tensor operations (what more than 1024 targets take), at
the edges of their blocks: one target, odd and even medians, a warp's and a block's worth of targets, the fewest
pulses the filter takes, histories of zeros.  Tolerance 1e-9 of the largest correction: FP64 sums of up to 2048
terms in another order (1e-13), through 2 x 2 solutions whose determinant the 0.002 regularisation bounds.

The spread section filter is compared bit for bit with the recursion in test_gpu_autofocus.py (two sections); here
one and three sections, and four (the cascade per lane).
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
    from bp_project_gb300 import _native
    return _native.load()


@pytest.mark.parametrize("targets,pulses", [(1, 64), (2, 20), (3, 601), (31, 100), (32, 503), (33, 504), (144, 700),
                                            (1023, 40), (1024, 64)])
def test_update_matches_the_tensor_operations(lib, monkeypatch, targets, pulses):
    from bp_project_gb300 import autofocus
    rng = np.random.default_rng(targets)
    pos = np.column_stack([rng.normal(0, 0.02, pulses), 0.1 * np.arange(pulses), np.full(pulses, 3000.0)])
    pts = np.column_stack([2700.0 + rng.uniform(0, 200, targets), rng.uniform(-100, 100, targets), np.zeros(targets)])
    data = torch.from_numpy((rng.standard_normal((pulses, 700)) + 1j * rng.standard_normal((pulses, 700)))
                            .astype(np.complex64)).cuda()
    args = (data, torch.from_numpy(pos).cuda(), torch.from_numpy(pts).cuda(), 3990.0, 0.8328, 402.0, 1000.0, 8.0)
    delta, stats = autofocus.estimate_update(*args)
    monkeypatch.setattr(lib, "sarbp_pga_max_targets", lambda: 0)
    want, wstats = autofocus.estimate_update(*args)
    top = float(want.abs().max())
    assert top > 0 and float((delta - want).abs().max()) <= 1e-9 * top
    assert stats.keys() == wstats.keys()
    for key in ("median_gradient_coherence", "delta_rms_m", "delta_max_m"):
        assert np.allclose(stats[key], wstats[key], rtol=1e-9, atol=1e-12 * top), key


def test_histories_of_zeros(lib, monkeypatch):
    from bp_project_gb300 import autofocus
    pos = np.column_stack([np.zeros(50), 0.1 * np.arange(50), np.full(50, 3000.0)])
    args = (torch.zeros((50, 300), dtype=torch.complex64, device="cuda"), torch.from_numpy(pos).cuda(),
            torch.tensor([[2700.0, 0.0, 0.0], [2710.0, 5.0, 0.0]], dtype=torch.float64, device="cuda"), 3990.0, 0.8328,
            402.0, 1000.0, 8.0)
    delta, _ = autofocus.estimate_update(*args)
    monkeypatch.setattr(lib, "sarbp_pga_max_targets", lambda: 0)
    want, _ = autofocus.estimate_update(*args)
    assert torch.equal(delta.isnan(), want.isnan()) and torch.equal(delta.nan_to_num(), want.nan_to_num())


@pytest.mark.parametrize("order", [1, 2, 5, 6, 8])
def test_section_counts(lib, order):
    from scipy import signal
    from bp_project_gb300.autofocus import SmoothingFilter, sosfiltfilt
    rng = np.random.default_rng(order)
    sos = np.ascontiguousarray(signal.butter(order, 0.2, output="sos"))
    x = (rng.standard_normal((5, 97)) + 1j * rng.standard_normal((5, 97))).astype(np.complex64)
    for pad in (0, 12):
        f = SmoothingFilter(sos, np.ascontiguousarray(signal.sosfilt_zi(sos)), pad)
        ref = signal.sosfiltfilt(sos, x, axis=1, padtype="odd", padlen=pad)
        out = sosfiltfilt(torch.from_numpy(x).cuda(), f).cpu().numpy()
        assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()
