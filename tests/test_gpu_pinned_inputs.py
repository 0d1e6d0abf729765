"""tdbem_md_march from pinned host buffers with input copies that lag behind
the march (TDBEM_INPUT_DELAY holds every chunk after the first back): each
history pass has to wait for the prescribed values of the steps it covers, up to
two passes ahead of the marched one.  The device buffer holds another call's
values before, so what is read early shows; the results must equal the march
from pageable buffers bit for bit.
"""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loads,n,nstep,env", [
    (1, 3, 30, {"TDBEM_RUNS": "2"}),                                # rows pass, a part beside each step
    (1, 3, 40, {"TDBEM_RUNS": "2", "TDBEM_HISTORY_STEPS": "3"}),
    (1, 3, 40, {"TDBEM_RUNS": "0"}),                                # one-step pass
    (1, 3, 20, {"TDBEM_RUNS": "2", "TDBEM_OVERLAP": "0"}),          # passes on the chain stream
    (4, 3, 31, {}),                                                 # run layout
    (8, 3, 30, {}),                                                 # group layout
    (8, 3, 64, {"TDBEM_HISTORY_STEPS": "3"}),                       # chunks of two and three steps
])
def test_late_input_copies(loads, n, nstep, env):
    import torch
    from tdbem import cases
    from tdbem.api import MultiDomainSolver, Report, load_library
    c = cases.config_bar8_batched(nstep=nstep, n=n, loads=loads, error=1e-12)
    # every element's prescribed values differ from step to step
    c.known += np.random.default_rng(5).normal(size=c.known.shape)
    old = {k: os.environ.get(k) for k in [*env, "TDBEM_INPUT_DELAY"]}
    os.environ.update(env)
    try:
        s = MultiDomainSolver(c, n_loads=loads)
        s.assemble()
        lu0, lt0, _ = s.march(c.known)
        s.march(-3.0 * c.known)
        kh = torch.from_numpy(np.ascontiguousarray(c.known)).pin_memory()
        lu, lt = torch.zeros_like(kh).pin_memory(), torch.zeros_like(kh).pin_memory()
        rep = Report()
        os.environ["TDBEM_INPUT_DELAY"] = "2000"
        assert load_library().tdbem_md_march(s.h, ctypes.c_void_p(kh.data_ptr()), ctypes.c_void_p(lu.data_ptr()),
                                             ctypes.c_void_p(lt.data_ptr()), ctypes.byref(rep), None) == 0
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.update({k: v})
    s.close()
    assert rep.steps_solved == nstep
    assert np.array_equal(lu.numpy(), lu0) and np.array_equal(lt.numpy(), lt0)
