"""Range compression by overlap-save blocks (oversample 1) against the same correlation in FP64, at the
edges of its range: fewer samples than taps, one output more or less than a block gives, odd
lengths (rows that start off a 16-byte boundary), the longest pulse that fits and one that does not
(the FFT steps), one tap's worth of filter and the most taps.

Tolerance 2e-6: two 2048-point FP32 transforms of eleven radix-2 stages each, sqrt(22) roundings of 6e-8
on average (3e-7), with room for the filter spectrum's own rounding.  (Pulses of a few samples are left out: their output is a
cancelling difference of neighbouring taps, 1e-5 off by conditioning alone in any FP32 transform.)
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
    from bp_project_gb300 import _native
    return _native.load()


def correlate64(raw, h):
    x = raw.astype(np.complex128)
    x = x - x.mean(axis=1, keepdims=True)
    n, first = len(h), len(h) - 1 - len(h) // 2
    size = x.shape[1] + n - 1
    full = np.fft.ifft(np.fft.fft(x, n=size, axis=1) * np.fft.fft(h.astype(np.complex128), n=size), axis=1)
    return full[:, first:first + x.shape[1]]


@pytest.mark.parametrize("pulses,samples,tp", [(3, 399, 1e-6), (2, 1649, 1e-6), (5, 1650, 1e-6),
                                               (3, 3299, 1e-6), (700, 1001, 1e-6), (4, 24576, 1e-6),
                                               (2, 24577, 1e-6), (3, 5000, 2.5e-9), (3, 2049, 1025 / 400e6),
                                               (2, 3000, 1026 / 400e6)])
def test_blocks_match_the_fp64_correlation(lib, pulses, samples, tp):
    from bp_project_gb300 import sar_io
    rng = np.random.default_rng(samples)
    raw = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples)) + (3 - 2j))
    raw = raw.astype(np.complex64)
    h = sar_io.matched_filter(tp, 200e6, -1)
    fits = bool(lib.sarbp_rc_blocks_fit(samples, len(h)))
    assert fits == (samples <= 24576 and len(h) <= 1025)
    out = sar_io.range_compress(torch.from_numpy(raw).cuda(), tp=tp).cpu().numpy()
    err = rel_err(correlate64(raw, h), out)
    assert err <= 2e-6, err


def test_a_value_that_is_not_finite_stays_in_its_pulse(lib):
    from bp_project_gb300 import sar_io
    rng = np.random.default_rng(0)
    raw = (rng.standard_normal((4, 2500)) + 1j * rng.standard_normal((4, 2500))).astype(np.complex64)
    clean = sar_io.range_compress(raw)
    raw[1, 77], raw[2, 2499] = np.nan, np.inf
    out = sar_io.range_compress(raw)
    assert np.array_equal(out[[0, 3]], clean[[0, 3]])
    assert np.isnan(out[1]).all() and not np.isfinite(out[2]).any()


def test_blocks_reject_what_does_not_fit(lib):
    import ctypes
    from bp_project_gb300 import _native
    fake = ctypes.c_void_p(0x10000)
    assert lib.sarbp_rc_blocks(fake, 0, 100, 40, fake, fake, None) == _native.SARBP_ERR_VALUE
    assert lib.sarbp_rc_blocks(fake, 4, 24577, 40, fake, fake, None) == _native.SARBP_ERR_VALUE
    assert lib.sarbp_rc_blocks(fake, 4, 100, 1026, fake, fake, None) == _native.SARBP_ERR_VALUE
    assert lib.sarbp_rc_blocks(None, 4, 100, 40, fake, fake, None) == _native.SARBP_ERR_TYPE
