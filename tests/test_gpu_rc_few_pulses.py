"""Range compression in one kernel with fewer pulses than SMs and a large offset (forty times the noise), against the same
correlation in FP64: a single pulse of one sample more than a block's outputs, of many blocks, and of the most samples.
A mean a last bit off leaves 3.8e-6 of offset in its pulse, which the filter's sum of taps carries to the output.

Tolerance 2e-6, as for the other lengths: two 2048-point FP32 transforms.
"""
import numpy as np
import pytest

from conftest import rel_err

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pulses,samples", [(1, 1650), (1, 8192), (1, 24576), (2, 24575), (151, 3300)])
def test_few_pulses(pulses, samples):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from bp_project_gb300 import build, sar_io
    build.build()
    rng = np.random.default_rng(samples)
    raw = rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples)) + (40 - 15j)
    raw = raw.astype(np.complex64)
    h = sar_io.matched_filter(1e-6, 200e6, -1)
    n = len(h)
    x = raw.astype(np.complex128)
    x -= x.mean(axis=1, keepdims=True).astype(np.complex64)  # the mean is taken off as a complex64 value
    size, first = samples + n - 1, n - 1 - n // 2
    full = np.fft.ifft(np.fft.fft(x, n=size, axis=1) * np.fft.fft(h.astype(np.complex128), n=size), axis=1)
    out = sar_io.range_compress(torch.from_numpy(raw).cuda()).cpu().numpy()
    assert rel_err(full[:, first:first + samples], out) <= 2e-6
