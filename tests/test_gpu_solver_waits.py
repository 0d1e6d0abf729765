"""A wait of the GMRES cluster that runs out fails the step: the call returns the
failure status with the step's number, nothing hangs, and the handle serves the
next call as before (B200).

TDBEM_GMRES_WAIT = -w (w >= 0) makes the last thread of the last CTA give up its
first wait, which no other thread of its CTA notices, and lets all further waits
run out after 2^w cycles; in the shared-memory and the global-memory form of the
kernel.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _with(env, call):
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        return call()
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.update({k: v})


@pytest.mark.parametrize("loads,precision,dsm,limit", [
    (1, "fp64", "1", "0"), (1, "fp64", "0", "-21"), (1, "mixed", "1", "-21"),
    (4, "mixed", "0", "0"), (8, "fp64", "1", "-21"), (32, "mixed", "1", "0"),
])
def test_wait_that_runs_out_fails_the_step(loads, precision, dsm, limit):
    from tdbem import cases
    from tdbem.api import MultiDomainSolver
    c = cases.config_rod5_batched(nstep=9, n=3, loads=loads, error=1e-11)
    s = MultiDomainSolver(c, precision=precision, n_loads=loads)
    s.assemble()
    form = {"TDBEM_GMRES_DSM": dsm}
    lu, lt, rep = _with(form, lambda: s.march(c.known))
    assert rep.steps_solved == c.nstep
    _, _, bad = _with({**form, "TDBEM_GMRES_WAIT": limit}, lambda: s.march(c.known, raise_on_failure=False))
    assert (bad.failed_step, bad.gmres_flag, bad.steps_solved) == (1, 1, 0)
    lu1, lt1, rep = _with(form, lambda: s.march(c.known))
    s.close()
    assert rep.steps_solved == c.nstep and np.array_equal(lu, lu1) and np.array_equal(lt, lt1)


def test_bare_solve():
    import torch
    from tdbem import cases
    from tdbem.api import MultiDomainSolver, TdbemError
    c = cases.config_rod5_batched(nstep=2, n=3, loads=1, error=1e-11)
    s = MultiDomainSolver(c)
    s.assemble()
    b = torch.randn(3 * c.n_elements, dtype=torch.float64, device="cuda")
    x, y = torch.zeros_like(b), torch.zeros_like(b)
    s.solve_noalloc(b.data_ptr(), x.data_ptr())
    with pytest.raises(TdbemError, match="GMRES flag 1"):
        _with({"TDBEM_GMRES_WAIT": "0"}, lambda: s.solve_noalloc(b.data_ptr(), y.data_ptr()))
    s.solve_noalloc(b.data_ptr(), y.data_ptr())
    s.close()
    assert torch.equal(x, y)
