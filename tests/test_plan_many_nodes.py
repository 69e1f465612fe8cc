"""The planner works on all nodes at once; every number equals the one-by-one planner's."""
import numpy as np
import pytest

from bp_project_gb300 import core
from bp_project_gb300 import gpu_backend as gb
from oracle.plan import plan_ffbp


@pytest.mark.parametrize("pulses,leaf,side,along", [(1, 64, 1, 1), (2, 1, -1, 1), (17, 16, 1, 0), (129, 3, -1, 1),
                                                    (1024, 64, 1, 1), (1500, 33, 1, 0)])
def test_equals_one_by_one(pulses, leaf, side, along):
    rng = np.random.default_rng(pulses)
    pos = rng.normal(0.0, 0.05, (pulses, 3)) + [0.0, 0.0, 3000.0]
    pos[:, along] += 0.1 * (np.arange(pulses) - pulses / 2) * (1.0 if along else 0.2)
    args = (pos, 9.6e9, (4000.0, 4210.0, -0.05, 0.07), side, leaf, 0.25, 2.5)
    want, plan = plan_ffbp(*args), gb.build_ffbp_plan(*args)
    nodes = plan.nodes()
    table = core.node_array(nodes)
    assert len(want.nodes) == len(nodes) == len(table)
    assert want.crop_r == plan.crop_r and want.crop_u == plan.crop_u
    assert {k: plan.counts[k] for k in want.counts} == want.counts
    for w, n, t in zip(want.nodes, nodes, table):
        assert np.array_equal(w.origin, n.origin) and list(t.origin) == list(w.origin)
        for name in ("r0", "dr", "u0", "du", "nr", "nu", "a", "b", "side"):
            assert getattr(w, name) == getattr(n, name) == getattr(t, name), name
        assert (w.left, w.right) == (t.left, t.right)
