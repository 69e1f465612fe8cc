"""Trajectory updates in which something is no number, against the tensor operations (a sort takes it for the largest value):
a target whose history is zero has no coherence, a sample that is no number spoils the targets that meet it.

Tolerance 1e-9, as for the other updates: FP64 sums in another order.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def both(monkeypatch, data, targets, k=402.0):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import _native, autofocus, build
    build.build()
    pulses = len(data)
    pos = np.column_stack([np.zeros(pulses), 0.1 * np.arange(pulses), np.full(pulses, 3000.0)])
    args = (*(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, targets)), 3990.0, 0.8328, k, 1000.0,
            8.0)
    found = autofocus.estimate_update(*args)
    monkeypatch.setattr(_native.load(), "sarbp_pga_max_targets", lambda: 0)
    return found, autofocus.estimate_update(*args)


def compare(found, want):
    (delta, stats), (wdelta, wstats) = found, want
    assert np.allclose(delta.cpu().numpy(), wdelta.cpu().numpy(), rtol=1e-9, equal_nan=True)
    for key in ("median_gradient_coherence", "delta_rms_m", "delta_max_m"):
        assert np.allclose(stats[key], wstats[key], rtol=1e-9, equal_nan=True), (key, stats[key], wstats[key])


def scene(targets, outside):
    rng = np.random.default_rng(targets)
    data = (rng.standard_normal((50, 300)) + 1j * rng.standard_normal((50, 300))).astype(np.complex64)
    pts = np.column_stack([2700.0 + rng.uniform(0, 100, targets), rng.uniform(-20, 20, targets), np.zeros(targets)])
    pts[:outside, 0] = 9000.0  # beyond the last bin
    return data, pts


@pytest.mark.parametrize("targets,outside", [(2, 1), (3, 1), (5, 2), (6, 5), (4, 4)])
def test_targets_without_a_history(monkeypatch, targets, outside):
    compare(*both(monkeypatch, *scene(targets, outside)))


@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf])
def test_samples_that_are_no_numbers(monkeypatch, value):
    data, pts = scene(7, 0)
    data[20, :60] = value
    compare(*both(monkeypatch, data, pts))


def test_without_a_wavenumber(monkeypatch):
    """k = 0: gradients have no length, so the corrections are no numbers; the call is taken all the same."""
    found, want = both(monkeypatch, *scene(5, 0), k=0.0)
    assert bool(want[0][:, :2].isnan().all())
    compare(found, want)
