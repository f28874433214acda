"""Grid barrier on one growing 32-bit counter: whether an observed count
completes a goal must not depend on where the counter wraps.  The comparison of
isl_device.cuh, restated, over a barrier of every position around the wrap."""
import os
import re

import numpy as np
import pytest

from conftest import ROOT


@pytest.mark.parametrize("ctas", [1, 2, 31, 152])
def test_goal_is_met_by_the_last_arrival_only(ctas):
    with open(os.path.join(ROOT, "insilico_gb300", "csrc", "isl_device.cuh")) as f:
        body = f.read().split("struct GridBarrier", 1)[1]
    cond = re.search(r"if \((.*)\) break;", body).group(1)
    expr = {"v >= goal": lambda v, g: v >= g,
            "(int)(v - goal) >= 0": lambda v, g: (v - g).astype(np.int32) >= 0}[cond]
    for start in list(range(2 ** 32 - 2 * ctas - 1, 2 ** 32)) + [0, 1, 2 ** 31 - ctas, 2 ** 31]:
        goal = np.uint32((start + ctas) % 2 ** 32)
        # from the first arrival of this barrier up to all of the next one's
        seen = ((start + 1 + np.arange(2 * ctas, dtype=np.uint64)) % 2 ** 32).astype(np.uint32)
        with np.errstate(over="ignore"):
            met = expr(seen, goal)
        assert not met[:ctas - 1].any() and met[ctas - 1:].all()
