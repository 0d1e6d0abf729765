"""The T-step history pass of one load case over the step-major matrices against
the one-step pass (B200): both precisions, T = 2 and 3, marches shorter than the
history and ending inside a pass, and the shortest history that takes it.

Both compute the sums of DBEM1/multidomain.cpp:3843-3866 in another order.
FP64 rounding of some 1,000 terms per sum over 30 steps stays under 1e-12 of the
largest value; the mixed march is held to 1e-8 at its tolerance of 1e-12, as its
FP32 Krylov spaces differ.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _march(case, precision, env):
    from tdbem.api import MultiDomainSolver
    os.environ.update(env)
    try:
        s = MultiDomainSolver(case, precision=precision)
        s.assemble()
    finally:
        for k in env:
            os.environ.pop(k)
    lu, lt, rep = s.march(case.known[0])
    s.close()
    assert rep.failed_step == 0
    return lu, lt, rep


@pytest.mark.parametrize("precision,mark", [("fp64", 1e-12), ("mixed", 1e-8)])
@pytest.mark.parametrize("n,nstep,beta,steps", [(3, 30, None, "2"), (3, 31, None, "3"), (4, 9, None, "2"), (4, 8, None, "3"),
                                                (1, 40, 0.1, "2"), (2, 21, 0.6, "3"), (1, 12, 0.9, "2")])
def test_rows_pass_equals_one_step(n, nstep, beta, steps, precision, mark):
    from tdbem import cases
    c = cases.config_bar8(nstep=nstep, n=n, error=1e-12 if precision == "mixed" else 1e-13)
    if beta:
        c.beta = beta
    a = _march(c, precision, {"TDBEM_RUNS": "2", "TDBEM_HISTORY_STEPS": steps})
    b = _march(c, precision, {"TDBEM_RUNS": "0"})
    if b[2].history_steps >= 5:
        assert a[2].history_launches < b[2].history_launches
    for x, y in zip(a[:2], b[:2]):
        assert np.max(np.abs(x - y)) <= mark * np.max(np.abs(y))


@pytest.mark.parametrize("overlap", ["1", "0"])
def test_phase_times_add_up(overlap):
    """Head, GMRES and history times come from the device clock: on the chain, head
    and GMRES do not overlap (1 us of clock granularity a step and phase allowed)."""
    from tdbem import cases
    from tdbem.api import MultiDomainSolver
    c = cases.config_bar8(nstep=30, n=3)
    s = MultiDomainSolver(c)
    s.assemble()
    os.environ["TDBEM_OVERLAP"] = overlap
    try:
        rep = s.march(c.known[0])[2]
    finally:
        os.environ.pop("TDBEM_OVERLAP")
    head = rep.ms_rhs - rep.ms_history
    assert rep.ms_gmres > 0 and head > 0 and rep.ms_history > 0
    chain = rep.ms_gmres + head + (rep.ms_history if overlap == "0" else 0.0)
    assert chain <= rep.ms_total + 3e-3 * c.nstep
