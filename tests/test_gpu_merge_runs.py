"""FFBP merge tiles (runs of eight rows per thread, expanded about their middle) where the expansion, the
tile edges and the fallbacks can go wrong: one merge of two supplied images against the FP64 regridding.

Tolerance 1e-5: the split policy's bound.  Range places are exact to 1e-7 bins, angle places (up to 16 bins
from the tile's centre in FP32) to 2e-6, phases to 3e-7 turns, and the FP32 sums add about 1e-6.
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


CASES = {
    # name: r0, dr, nr, u0, du, nu, side, origins' distance (x, y, z), child's row and column steps / the parent's
    "deep_level": (4000.3, 0.25, 133, -0.1, 2e-3, 75, 1, (0.0, 1.6, 0.0), 1.0, 2.0),
    "root_level": (4000.3, 0.25, 71, 0.05, 1.5e-5, 333, 1, (0.3, 204.8, 0.2), 1.0, 2.0),
    "left_curved": (4400.0, 0.3, 40, -0.3, 2e-4, 60, -1, (4.0, 20.0, -1.0), 1.0, 2.0),
    "one_pixel": (4000.3, 0.25, 1, 0.1, 1e-3, 1, 1, (0.0, 3.2, 0.0), 1.0, 2.0),
    "other_rows": (4000.3, 0.25, 50, -0.02, 1e-3, 40, 1, (0.0, 3.2, 0.0), 1.6, 1.3),
    "near_nadir": (3004.0, 0.25, 64, 0.0, 1e-3, 40, 1, (0.0, 12.8, 0.0), 1.0, 2.0),       # pair by pair
}


@pytest.mark.parametrize("name", CASES)
def test_merge_matches_the_fp64_regridding(lib, name):
    from bp_project_gb300 import core
    from bp_project_gb300.gpu_backend import NodePlan
    from oracle import reference as ora
    r0, dr, nr, u0, du, nu, side, apart, fr, fu = CASES[name]
    rng = np.random.default_rng(len(name))
    origin, k = np.array([5.0, -3.0, 3000.0]), 402.0
    nodes, images, ref = [NodePlan(0, 0, 2, origin, r0, dr, nr, u0, du, nu, side)], [], 0.0
    for c in (-1, 1):
        o = origin + 0.5 * c * np.array(apart)
        # The parent's corners seen from the child, and a border of which some pixels' stencils stay outside.
        r, u = np.meshgrid(r0 + dr * np.linspace(0, nr - 1, 9), u0 + du * np.linspace(0, nu - 1, 9))
        g = np.sqrt(r * r - origin[2] ** 2)
        x, y = origin[0] + side * g * np.sqrt(1 - u * u) - o[0], origin[1] + g * u - o[1]
        gc = np.hypot(x, y)
        rc, uc = np.sqrt(gc * gc + o[2] ** 2), y / gc
        sdr, sdu = fr * dr, fu * du
        sr0, su0 = rc.min() - 2.4 * sdr, uc.min() - 0.6 * sdu
        snr, snu = int((rc.max() - sr0) / sdr) + 4, int((uc.max() - su0) / sdu) + 4
        img = (rng.standard_normal((snr, snu)) + 1j * rng.standard_normal((snr, snu))).astype(np.complex64)
        ref = ref + ora.regrid(img, o, sr0, sdr, su0, sdu, origin, r0, dr, nr, u0, du, nu, k, side, c128=True)[1]
        nodes.append(NodePlan(len(nodes), -1, -1, o, sr0, sdr, snr, su0, sdu, snu, side))
        images.append(torch.from_numpy(img).cuda())
    nodes[0].left, nodes[0].right = nodes[1], nodes[2]
    data = torch.zeros((2, 16), dtype=torch.complex64, device="cuda")
    pos, one = torch.zeros((2, 3), dtype=torch.float64, device="cuda"), torch.ones(2, dtype=torch.float64, device="cuda")
    out = []
    for opts in ({}, {"staging": False}, {"merge_queue": True}):
        program = core.FFBPProgram(nodes, (0, nr), (0, nu), **opts)
        for n, img in enumerate(images):
            program.set_node_image(n + 1, img)
        out.append(program.execute(data, pos, one, one, 0.0, 0.8327, k).cpu().numpy())
        torch.cuda.synchronize()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    assert np.linalg.norm(out[0] - ref) <= 1e-5 * np.linalg.norm(ref), name
