"""Which form of the T-step history pass a handle takes (B200), told by the report:
a launch of the group form loads a history vector for 8 rows and two steps at
once, so its loads stay under a third of the block steps; the run and rows forms
load at least 0.6 of them; the one-step pass is launched every step.
"""
import os

import numpy as np
import pytest

from test_gpu_nonfinite import _case, _march, _matrices

pytestmark = pytest.mark.gpu

K, NSTEP = 14, 25


@pytest.mark.parametrize("loads,share,runs,form", [
    (8, 0.5, "1", "groups"), (32, 0.5, "1", "groups"),
    (8, 0.02, "1", "runs"),   # a group's fragments would be filled to 2 * 0.02 of 0.4
    (4, 0.5, "1", "runs"), (2, 0.5, "1", "runs"),
    (1, 0.5, "2", "rows"), (1, 0.5, "1", "one step"),  # 126 MB of blocks or TDBEM_RUNS=2
    (8, 0.5, "0", "one step"),
])
def test_form_by_report(loads, share, runs, form):
    c = _case(loads, NSTEP)
    rep = _march(c, loads, "fp64", _matrices(c.n_elements, K, share), TDBEM_RUNS=runs)[2]
    assert rep.steps_solved == NSTEP
    ratio = rep.history_vector_loads / rep.history_block_steps
    assert rep.history_launches == (NSTEP - 2 if form == "one step" else (NSTEP - 3 + 1) // 2)
    if form == "one step":
        assert ratio == 1.0
    elif form == "groups":
        assert ratio < 1 / 3
    else:
        assert ratio > 0.6
