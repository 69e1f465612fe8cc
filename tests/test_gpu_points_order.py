"""Point lists in spatial order (split-mode direct BP at points): raster, shuffled, clustered and degenerate lists
against the FP64 oracle, at the edges of a tile (1024 points) and of a sorting block (4096), with and without the
workspace that the order needs, repeated bit for bit, and captured in a graph.

Tolerance 1e-5: the split policy's bound.
"""
import ctypes

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


def scene(xyz, pulses=70, seed=0):
    rng = np.random.default_rng(seed)
    pos = np.column_stack([np.zeros(pulses), 0.1 * np.arange(pulses), np.full(pulses, 3000.0)])
    r = np.linalg.norm(xyz[None] - pos[::pulses - 1, None], axis=2)
    start, dr = float(r.min()) - 20.0, 0.8328
    samples = int((r.max() - start) / dr) + 20
    data = (rng.standard_normal((pulses, samples)) + 1j * rng.standard_normal((pulses, samples))).astype(np.complex64)
    return data, pos, rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses), start, dr, 402.0


def points(kind, n, rng):
    if kind == "raster":  # rows of 333 points half a metre apart, on hills
        i, j = np.divmod(np.arange(n), 333)
        xyz = np.column_stack([2700.0 + 0.5 * i, 0.5 * j, 3.0 * np.sin(0.05 * j)])
    elif kind == "shuffled":
        xyz = np.column_stack([2700.0 + rng.uniform(0, 40, n), rng.uniform(0, 40, n), rng.uniform(-1, 1, n)])
    elif kind == "patches":  # points around targets hundreds of metres apart
        c = rng.uniform(0, 600, (9, 2))[np.arange(n) * 9 // n]
        xyz = np.column_stack([2700.0 + c[:, 0] + rng.uniform(-3, 3, n), c[:, 1] + rng.uniform(-3, 3, n), np.zeros(n)])
    else:  # one line, every point twice
        xyz = np.column_stack([np.full(n, 2700.0), 0.3 * (np.arange(n) // 2), np.zeros(n)])
    return np.ascontiguousarray(xyz)


@pytest.mark.parametrize("n", [1024, 1025, 4096, 4097, 9001])
@pytest.mark.parametrize("kind", ["raster", "shuffled", "patches", "line"])
def test_point_lists_match_the_fp64_oracle(lib, kind, n):
    from bp_project_gb300 import core
    from oracle import reference as ora
    xyz = points(kind, n, np.random.default_rng(n))
    data, pos, w, ph, start, dr, k = scene(xyz)
    _, ref = ora.backproject_points(data, pos, xyz, start, dr, k, w, ph, c128=True)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, w, ph, xyz)]
    out = core.backproject_points(*args, start, dr, k)
    assert rel_err(ref, out.cpu().numpy()) <= 1e-5
    assert torch.equal(out, core.backproject_points(*args, start, dr, k))
    split = core.backproject_points(*args, start, dr, k, pulse_split=3)
    assert rel_err(ref, split.cpu().numpy()) <= 1e-5


def test_without_the_workspace_and_captured(lib):
    from bp_project_gb300 import _native as nat
    from bp_project_gb300 import core
    xyz = points("raster", 5000, np.random.default_rng(1))
    data, pos, w, ph, start, dr, k = scene(xyz)
    args = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (data, pos, w, ph, xyz)]
    want = core.backproject_points(*args, start, dr, k)
    plain = torch.empty_like(want)
    p, s = data.shape
    call = [core._ptr(args[0]), p, s, *(core._ptr(a) for a in args[1:]), 5000, start, dr, k, nat.MODE_IDS["split"]]
    assert lib.sarbp_backproject_points(*call, 1, core._ptr(plain), None, 0, core.stream_handle()) == nat.SARBP_OK
    assert rel_err(want.cpu().numpy(), plain.cpu().numpy()) <= 1e-5
    part = torch.empty(3 * 5000 * 8, dtype=torch.uint8, device="cuda")  # the partial images alone
    assert lib.sarbp_backproject_points(*call, 3, core._ptr(plain), core._ptr(part), part.numel(),
                                        core.stream_handle()) == nat.SARBP_OK
    assert rel_err(want.cpu().numpy(), plain.cpu().numpy()) <= 1e-5
    assert lib.sarbp_backproject_points(*call, 3, core._ptr(plain), core._ptr(part), part.numel() - 1,
                                        core.stream_handle()) == nat.SARBP_ERR_WORKSPACE
    out = torch.zeros_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        core.backproject_points(*args, start, dr, k, out=out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
