"""CudaBaseline.kernel_names: every name is a kernel of the sources, and the kernels that run_direct and run_ffbp launch
are among them."""
import re
from pathlib import Path

from bp_project_gb300 import gpu_backend


def test_names_are_kernels_of_the_sources():
    csrc = Path(gpu_backend.__file__).resolve().parent / "csrc"
    kernels = set()
    for path in csrc.glob("*.cu"):
        kernels |= set(re.findall(r"(\w+_kernel)\(", path.read_text()))
    names = [n.split("<")[0] for n in gpu_backend.CudaBaseline.kernel_names]
    assert set(names) <= kernels and len(names) == len(set(names))
    launched = {"split_polar_kernel", "split_polar_runs_kernel", "split_leaf_kernel", "split_merge_kernel",
                "split_merge_staged_kernel", "plain_polar_kernel", "plain_ffbp_leaf_kernel", "plain_ffbp_merge_kernel"}
    assert launched <= set(names)
