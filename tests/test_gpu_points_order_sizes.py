"""Spatial order of point lists at the sizes where its passes can go wrong, against the FP64 oracle: a tile (512 points) and
one more, a counting block's round of 256 keys, lists at which the blocks (one per SM, 152) begin to take two rounds
and a remainder, and a compact list, which is taken as it is.

Tolerance 1e-5: the split policy's bound.
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


def scene(xyz, pulses):
    rng = np.random.default_rng(len(xyz))
    pos = np.column_stack([np.zeros(pulses), 0.1 * np.arange(pulses), np.full(pulses, 3000.0)])
    r = np.linalg.norm(xyz[None] - pos[[0, -1], None], axis=2)
    start, dr = float(r.min()) - 20.0, 0.8328
    samples = int((r.max() - start) / dr) + 20
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    return (data, pos, rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses)), (start, dr, 402.0)


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("n", [511, 512, 513, 767, 769, 24064, 24065, 38912, 38913, 60001])
def test_sizes(lib, n, shuffled):
    from bp_project_gb300 import core
    from oracle import reference as ora
    i, j = np.divmod(np.arange(n), 333)
    xyz = np.column_stack([2700.0 + 0.5 * i, 0.5 * j, 3.0 * np.sin(0.05 * j)])
    if shuffled:
        xyz = np.ascontiguousarray(xyz[np.random.default_rng(n).permutation(n)])
    arrays, radar = scene(xyz, 6)
    data, pos, w, ph = arrays
    _, ref = ora.backproject_points(data, pos, xyz, *radar, w, ph, c128=True)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (*arrays, xyz)]
    out = core.backproject_points(*args, *radar, pulse_split=1)
    assert rel_err(ref, out.cpu().numpy()) <= 1e-5
    assert torch.equal(out, core.backproject_points(*args, *radar, pulse_split=1))


@pytest.mark.parametrize("n", [513, 1300, 5000])
def test_compact_lists_are_taken_as_they_are(lib, n):
    from bp_project_gb300 import _native as nat
    from bp_project_gb300 import core
    from oracle import reference as ora
    i, j = np.divmod(np.arange(n), 40)
    xyz = np.column_stack([2700.0 + 0.1 * i, 0.1 * j, np.zeros(n)])
    arrays, radar = scene(xyz, 20)
    data, pos, w, ph = arrays
    _, ref = ora.backproject_points(data, pos, xyz, *radar, w, ph, c128=True)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (*arrays, xyz)]
    out = core.backproject_points(*args, *radar, pulse_split=1)
    assert rel_err(ref, out.cpu().numpy()) <= 1e-5
    plain = torch.empty_like(out)
    assert lib.sarbp_backproject_points(core._ptr(args[0]), *data.shape, *(core._ptr(a) for a in args[1:]), n, *radar,
                                        nat.MODE_IDS["split"], 1, core._ptr(plain), None, 0,
                                        core.stream_handle()) == nat.SARBP_OK
    assert torch.equal(out, plain)


def test_wide_lists_at_a_far_range_are_ordered(lib):
    """At 30 km tiles of 33 m radius fit the fast path; ordered, they are compact, and the image is closer to FP64."""
    from bp_project_gb300 import _native as nat
    from bp_project_gb300 import core
    from oracle import reference as ora
    n = 68 * 266
    i, j = np.divmod(np.arange(n), 266)
    xyz = np.column_stack([3.0e4 + 0.25 * i, 0.25 * j, np.zeros(n)])
    arrays, radar = scene(xyz, 12)
    data, pos, w, ph = arrays
    _, ref = ora.backproject_points(data, pos, xyz, *radar, w, ph, c128=True)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (*arrays, xyz)]
    out = core.backproject_points(*args, *radar, pulse_split=1)
    plain = torch.empty_like(out)
    assert lib.sarbp_backproject_points(core._ptr(args[0]), *data.shape, *(core._ptr(a) for a in args[1:]), n, *radar,
                                        nat.MODE_IDS["split"], 1, core._ptr(plain), None, 0,
                                        core.stream_handle()) == nat.SARBP_OK
    assert rel_err(ref, out.cpu().numpy()) < rel_err(ref, plain.cpu().numpy()) <= 1e-5
