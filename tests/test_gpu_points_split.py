"""The pulse split of point lists: an explicit 1 is one pass over the pulses, 0 (the default) the library's choice, which
takes memory only where the split pays.

Sums are compared bit for bit where the passes are the same, and against each other within 1e-5 (the split policy's
bound) where they are not.
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


def scene(n, pulses):
    rng = np.random.default_rng(n)
    i, j = np.divmod(np.arange(n), 64)  # narrow as they come: taken in their own order
    xyz = np.column_stack([2700.0 + 0.2 * i, 0.2 * j, np.zeros(n)])
    pos = np.column_stack([np.zeros(pulses), 0.1 * np.arange(pulses), np.full(pulses, 3000.0)])
    data = (rng.standard_normal((pulses, 200)) + 1j * rng.standard_normal((pulses, 200))).astype(np.complex64)
    arrays = data, pos, rng.uniform(0.5, 1.5, pulses), rng.uniform(-3, 3, pulses), xyz
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays], (4020.0, 0.8328, 402.0)


@pytest.mark.parametrize("n,pulses", [(512, 9), (513, 40), (2000, 300)])
def test_one_pass_and_the_automatic_split(lib, n, pulses):
    from bp_project_gb300 import _native as nat
    from bp_project_gb300 import core
    args, radar = scene(n, pulses)
    one = core.backproject_points(*args, *radar, pulse_split=1)
    plain = torch.empty_like(one)
    call = [core._ptr(args[0]), pulses, 200, *(core._ptr(a) for a in args[1:]), n, *radar]
    split, fp64 = nat.MODE_IDS["split"], nat.MODE_IDS["fp64"]
    assert lib.sarbp_backproject_points(*call, split, 1, core._ptr(plain), None, 0, core.stream_handle()) == nat.SARBP_OK
    assert torch.equal(one, plain)
    auto = core.backproject_points(*args, *radar)
    assert torch.equal(auto, core.backproject_points(*args, *radar, pulse_split=0))
    assert rel_err(one.cpu().numpy(), auto.cpu().numpy()) <= 1e-5
    assert torch.equal(core.backproject_points(*args, *radar, mode="fp64"),
                       core.backproject_points(*args, *radar, mode="fp64", pulse_split=1))
    for mode, bad in ((split, -1), (split, pulses + 1), (fp64, 2)):
        assert lib.sarbp_backproject_points(*call, mode, bad, core._ptr(plain), None, 0, None) == nat.SARBP_ERR_VALUE


@pytest.mark.parametrize("n", [513, 8000, 200_000, 20_000_000, 50_000_000])
def test_memory(lib, n):
    from bp_project_gb300 import _native as nat
    split = nat.MODE_IDS["split"]
    order = 14 * n + 128 * 1024  # two 16-bit keys and two indices per point, rounding, at most 96 K of counts
    assert lib.sarbp_backproject_points_workspace(split, n, 1) <= order
    assert lib.sarbp_backproject_points_workspace(split, n, 4) <= order + 32 * n
    auto = lib.sarbp_backproject_points_workspace(split, n, 0)
    assert auto <= order + (64 * n if n < 10_000_000 else 0)  # twenty rounds of tiles gain less than a twentieth
    assert lib.sarbp_backproject_points_workspace(nat.MODE_IDS["fp64"], n, 0) == 0
