"""Two threads in one entry point, with calls whose kernels take different amounts of shared memory: every call
succeeds and gives what it gives alone, bit for bit (the library keeps no state per call, so there is no tolerance).
"""
import threading

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


def noise(*shape):
    gen = torch.Generator(device="cuda").manual_seed(shape[-1])
    return torch.complex(torch.randn(shape, device="cuda", generator=gen), torch.randn(shape, device="cuda", generator=gen))


def zeros(*shape):
    return torch.zeros(shape, dtype=torch.float64, device="cuda")


# Each returns a library call on buffers of its own, without Python work in between, its output and what it reads.
def compress(lib, size):
    raw, response, out = noise(2, size), noise(lib.sarbp_rc_block_points()), noise(2, size)
    args = (raw.data_ptr(), 2, size, 400, response.data_ptr(), out.data_ptr(), None)
    return lib.sarbp_rc_blocks, args, out, (raw, response)


def smooth(lib, size):
    from bp_project_gb300 import autofocus
    f = autofocus.butter_lowpass(8.0, 1000.0)
    x, out = noise(2, size), zeros(2, size, 2)
    sos, zi = torch.from_numpy(f.sos).cuda(), torch.from_numpy(f.zi).cuda()
    ws = zeros(lib.sarbp_sosfiltfilt_workspace(2, size, f.padlen) // 8 + 1)
    args = (x.data_ptr(), 2, size, sos.data_ptr(), zi.data_ptr(), len(f.sos), f.sos.ctypes.data, f.padlen, out.data_ptr(),
            ws.data_ptr(), ws.numel() * 8, None)
    return lib.sarbp_sosfiltfilt, args, out, (x, sos, zi, f, ws)


def update(lib, size):
    pos, pts = zeros(5, 3), zeros(size, 3)
    pos[:, 1], pos[:, 2] = 0.1 * torch.arange(5), 3000.0
    pts[:, 0] = 2700.0 + 0.05 * torch.arange(size)
    histories = noise(size, 5).to(torch.complex128)
    rows, out, stats = zeros(3, 3) + 1.0 / 3.0, zeros(5, 3), zeros(7)
    ws = zeros(lib.sarbp_pga_update_workspace(size, 5) // 8)
    r = rows.data_ptr()
    args = (histories.data_ptr(), size, 5, pos.data_ptr(), pts.data_ptr(), 402.0, r, r, r, 3, out.data_ptr(),
            stats.data_ptr(), ws.data_ptr(), ws.numel() * 8, None)
    return lib.sarbp_pga_update, args, out, (pos, pts, histories, rows, stats, ws)


def polar(lib, size):
    import ctypes

    from bp_project_gb300 import _native as nat
    from bp_project_gb300 import core
    pos, ones, zero = zeros(40, 3), zeros(40) + 1.0, zeros(40)
    pos[:, 1], pos[:, 2] = 0.1 * torch.arange(40), 3000.0
    data, out = noise(40, size), noise(64, 64)
    grid = core.Grid((0.0, 2.0, 3000.0), 4000.0, 0.25, 64, -0.02, 0.0004, 64).native()
    args = (data.data_ptr(), 40, size, pos.data_ptr(), ones.data_ptr(), zero.data_ptr(), ctypes.byref(grid), 3990.0,
            40.0 / size, 402.0, nat.MODE_IDS["split"], size // 10, 1, out.data_ptr(), None, 0, None)
    return lib.sarbp_direct_polar, args, out, (data, pos, ones, zero, grid)


# Sizes in samples, samples, targets and samples: the two of a pair need different amounts above 48 KB.
@pytest.mark.parametrize("make,sizes,times", [(compress, (2000, 24000), 20000), (smooth, (3500, 9000), 300),
                                              (update, (900, 1024), 5000), (polar, (60, 640), 5000)],
                         ids=["compress", "smooth", "update", "polar"])
def test_two_threads(lib, make, sizes, times):
    calls = [make(lib, s) for s in sizes]
    want = []
    for call, args, out, _ in calls:
        assert call(*args) == 0
        want.append(out.clone())
        out.zero_()
    torch.cuda.synchronize()
    refused = []
    start = threading.Barrier(2)

    def work(call, args):
        start.wait()
        refused.append(sum(call(*args) != 0 for _ in range(times)))

    threads = [threading.Thread(target=work, args=c[:2]) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert refused == [0, 0]
    assert all(torch.equal(c[2], w) for c, w in zip(calls, want))
