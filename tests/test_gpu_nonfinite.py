"""Values that are not finite stay where the sums put them (B200).

A history vector combines three states (2 X_s + X_{s-1} + X_{s-2}), so states near
the largest double make an infinite one.  It reaches the rows and steps that have
a block for it and no others: with the cases and blocks below the right-hand side
of one load case becomes infinite, which counts as solved by zero, and every other
load case is as without it.  Likewise a block that is not finite has no part in the
steps before its own.  The passes that pad rows or steps with zeros (groups of
rows, the packed head) must not multiply the padding by either.

The reference is the one-step pass of the same march (TDBEM_RUNS=0), bit for bit
up to rounding of some hundred terms (1e-12), or the same march without the block.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(loads, nstep, error=1e-13):
    from tdbem import cases
    rng = np.random.default_rng(8)
    c = cases.make_case("cube", 1, 3, [cases.Material(20.0, 0.25, 20.0)], 0.6, nstep,
                        [(1.0, (1.0, 0.0, 0.0), cases.heaviside(nstep))] * loads, error=error)
    c.known *= rng.uniform(0.5, 2.0, size=(loads, 1, 1, 1))
    return c


def _csr(E, mask, v):
    i, j = np.nonzero(mask)
    return np.searchsorted(i, np.arange(E + 1)).astype(np.int32), j.astype(np.int32), v(i, j).reshape(-1, 9)


def _matrices(E, K, share, first=None, lone=None):
    """Seeded matrices; history column `lone` has blocks from step `first` on only,
    in a third of the rows, and no known block."""
    rng = np.random.default_rng(9)
    eye = np.eye(E, dtype=bool)

    def random(scale, diag=0.0):
        return lambda i, j: scale * rng.normal(size=(len(i), 3, 3)) + diag * (i == j)[:, None, None] * np.eye(3)

    A = _csr(E, eye | (rng.uniform(size=(E, E)) < 0.05), random(0.05, 2.0))
    known = eye.copy()
    if lone is not None:
        known[:, lone] = False
    Km = _csr(E, known, random(0.1, 1.0))
    hist = []
    for _ in range(2):
        hist.append([])
        for k in range(1, K + 1):
            on = rng.uniform(size=(E, E)) < share
            if lone is not None:
                on[:, lone] = (k >= first) & (rng.uniform(size=E) < 0.3)
            hist[-1].append(_csr(E, on, random(0.02)))
    return [A, Km, *hist]


def _march(c, loads, precision, matrices, **env):
    from tdbem.api import MultiDomainSolver
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        s = MultiDomainSolver(c, precision=precision, n_loads=loads)
        s.load_matrices(*matrices)
        out = s.march(c.known, raise_on_failure=False)
        s.close()
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.update({k: v})
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("loads,K,nstep", [(8, 14, 25), (16, 11, 20), (32, 9, 17)])
def test_infinite_history_vector(loads, K, nstep, precision):
    c = _case(loads, nstep, 1e-12 if precision == "mixed" else 1e-13)
    lone = int(np.nonzero(c.bcid == 123)[0][0])
    m = _matrices(c.n_elements, K, 0.5, 6, lone)
    c.known[1, 2, lone, 0] = 1.7e308  # load case 1, step 2
    assert np.isfinite(c.known).all()
    got, ref = _march(c, loads, precision, m), _march(c, loads, precision, m, TDBEM_RUNS="0")
    assert ref[2].failed_step == 0 and ref[2].steps_solved == nstep
    assert got[2].failed_step == 0 and got[2].steps_solved == nstep
    assert got[2].history_launches < ref[2].history_launches
    assert got[2].history_vector_loads < got[2].history_block_steps / 3  # groups: a vector serves 8 rows and 2 steps
    mark = 1e-8 if precision == "mixed" else 1e-12
    for r in range(loads):
        for q in range(2):
            a, b = got[q][r], ref[q][r]
            if r != 1:
                assert np.max(np.abs(a - b)) <= mark * np.max(np.abs(b)), (r, q)
            else:
                assert np.array_equal(np.isfinite(a), np.isfinite(b))


@pytest.mark.parametrize("loads,precision,at,nstep,value,env", [
    (1, "fp64", 2, 1, np.inf, {}),                                 # packed head of the one-step pass
    (1, "mixed", 2, 1, 1e300, {}),                                 # infinite as FP32
    (1, "fp64", 4, 3, np.nan, {"TDBEM_RUNS": "2"}),                # packed head of the two-step pass
    (8, "fp64", 14, 13, np.inf, {}), (8, "mixed", 14, 13, 1e300, {}),  # fragments past the last sum's step
])
def test_block_that_is_not_finite(loads, precision, at, nstep, value, env):
    c = _case(loads, nstep, 1e-12 if precision == "mixed" else 1e-13)
    m = _matrices(c.n_elements, 14, 0.5)
    ref = _march(c, loads, precision, m, **env)
    assert ref[2].failed_step == 0 and ref[2].steps_solved == nstep
    assert loads == 1 or ref[2].history_vector_loads < ref[2].history_block_steps / 2  # groups
    for hist in m[2:]:
        hist[at - 1][2][7::11] = value
    got = _march(c, loads, precision, m, **env)
    assert got[2].failed_step == 0 and got[2].steps_solved == nstep
    mark = 1e-8 if precision == "mixed" else 1e-12
    for q in range(2):
        assert np.max(np.abs(got[q] - ref[q])) <= mark * np.max(np.abs(ref[q])), q


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("loads", [2, 4, 8, 32])
def test_infinite_right_hand_side_beside_others(loads, precision):
    """Load cases that share a GMRES cluster with one whose right-hand side is
    infinite, against every case in its own cluster."""
    nstep = 20
    c = _case(loads, nstep, 1e-12 if precision == "mixed" else 1e-13)
    lone = int(np.nonzero(c.bcid == 123)[0][0])
    m = _matrices(c.n_elements, 11, 0.5, 6, lone)
    c.known[1, 2, lone, 0] = 1.7e308
    got = _march(c, loads, precision, m, TDBEM_GMRES_GROUPS="1", TDBEM_RUNS="0")
    ref = _march(c, loads, precision, m, TDBEM_GMRES_GROUPS=str(loads), TDBEM_RUNS="0")
    assert (got[2].gmres_groups, ref[2].gmres_groups) == (1, loads)
    for out in (got, ref):
        assert out[2].failed_step == 0 and out[2].steps_solved == nstep and np.isfinite(out[1]).all()
    mark = 1e-8 if precision == "mixed" else 1e-12
    for r in range(loads):
        for q in range(2):
            s = slice(None) if r != 1 else slice(0, 7)  # case 1: up to the infinite sums
            a, b = got[q][r, s], ref[q][r, s]
            assert np.max(np.abs(a - b)) <= mark * np.max(np.abs(b)), (r, q)
