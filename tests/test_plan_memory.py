"""A plan of many nodes is made in little memory: its work arrays hold a few nodes at a time."""
import tracemalloc

import numpy as np

from bp_project_gb300.gpu_backend import build_ffbp_plan


def test_peak_of_a_plan_of_16383_nodes():
    n = 32768
    pos = np.column_stack([np.zeros(n), 0.1 * (np.arange(n) - 0.5 * n), np.full(n, 3000.0)])
    tracemalloc.start()
    plan = build_ffbp_plan(pos, 9.6e9, (4000.0, 4100.0, -0.02, 0.02), leaf_size=4)
    kept, peak = tracemalloc.get_traced_memory()
    tracemalloc.stop()
    assert len(plan.nodes()) == 16383
    # All nodes' views of the 516 boundary points would be 68 MB per array; 128 nodes' are 0.5.
    assert peak - kept <= 32e6, (peak, kept)
