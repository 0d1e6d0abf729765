"""The group form of the T-step history pass (8 or more load cases) against the
one-step pass (B200): domains whose rows do not fill their last group, every
load count and precision it serves, marches that end inside a pass, and given
matrices whose blocks come at scattered steps, so that segments are cut at gaps,
or share too little between rows for groups (then the run layout serves).

Both compute the sums of DBEM1/multidomain.cpp:3843-3866 in another order.
FP64 rounding of some 1,000 terms per sum over 30 steps stays under 1e-12 of the
largest value; the mixed march is held to 1e-8 at its tolerance of 1e-12, as its
FP32 Krylov spaces differ.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def _solver(case, precision, loads, runs, matrices=None):
    from tdbem.api import MultiDomainSolver
    old = os.environ.get("TDBEM_RUNS")
    os.environ["TDBEM_RUNS"] = runs
    try:
        s = MultiDomainSolver(case, precision=precision, n_loads=loads)
        if matrices is None:
            s.assemble()
        else:
            s.load_matrices(*matrices)
    finally:
        os.environ.pop("TDBEM_RUNS") if old is None else os.environ.update(TDBEM_RUNS=old)
    return s


def _compare(case, precision, loads, mark, matrices=None):
    out = []
    for runs in ("1", "0"):
        s = _solver(case, precision, loads, runs, matrices)
        lu, lt, rep = s.march(case.known)
        s.close()
        assert rep.failed_step == 0
        out.append((lu, lt, rep))
    assert out[0][2].history_launches < out[1][2].history_launches
    for r in range(loads):
        assert _rel(out[0][0][r], out[1][0][r]) <= mark, r
        assert _rel(out[0][1][r], out[1][1][r]) <= mark, r


@pytest.mark.parametrize("precision,mark", [("fp64", 1e-12), ("mixed", 1e-8)])
@pytest.mark.parametrize("loads,n,nstep", [(8, 3, 29), (16, 3, 30), (32, 3, 31), (16, 5, 24), (8, 1, 12)])
def test_groups_equal_one_step(loads, n, nstep, precision, mark):
    from tdbem import cases
    c = cases.config_bar8_batched(nstep=nstep, n=n, loads=loads, error=1e-12 if precision == "mixed" else 1e-13)
    if n == 1:  # one element a face: make the history long with a small time step
        c.beta = 0.1
    _compare(c, precision, loads, mark)


@pytest.mark.parametrize("share", [0.02, 0.5])
def test_scattered_blocks(share):
    """Blocks at random steps; with a share of 0.02 of the (row, column, step)
    triples a group of 8 rows fills an eighth of its matrices."""
    from tdbem import cases
    rng = np.random.default_rng(8)
    loads, K, nstep = 8, 14, 25
    c = cases.make_case("cube", 1, 3, [cases.Material(20.0, 0.25, 20.0)], 0.6, nstep,
                        [(1.0, (1.0, 0.0, 0.0), cases.heaviside(nstep))] * loads, error=1e-13)
    c.known *= rng.uniform(0.5, 2.0, size=(loads, 1, 1, 1))
    E = c.n_elements

    def csr(mask, scale, diag=0.0):
        i, j = np.nonzero(mask)
        v = scale * rng.normal(size=(len(i), 3, 3))
        v[i == j] += diag * np.eye(3)
        return np.searchsorted(i, np.arange(E + 1)).astype(np.int32), j.astype(np.int32), v.reshape(-1, 9)

    eye = np.eye(E, dtype=bool)
    A = csr(eye | (rng.uniform(size=(E, E)) < 0.05), 0.05, 2.0)
    Km = csr(eye, 0.1, 1.0)
    hist = [[csr(rng.uniform(size=(E, E)) < share, 0.02) for _ in range(K)] for _ in range(2)]
    _compare(c, "fp64", loads, 1e-12, (A, Km, hist[0], hist[1]))
