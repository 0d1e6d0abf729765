"""The GMRES cluster kernel on its own, over its forms and sizes (B200).

One step of a cube without interfaces whose matrices are given: A x = K known,
against a dense solve.  Covered: load cases per cluster from 1 to 32, vectors in
shared memory and in global memory (TDBEM_GMRES_DSM=0), a single CTA, ranges of
uneven size, and more Krylov columns than the shared-memory arrays hold (the
block-diagonal preconditioner of one-element leaves leaves a spectrum of radius
about 0.65 around 1, some 60 steps to 1e-12).

Bound: the residual is at most tol |b|, so the error is at most tol cond(A) |x|
in the 2-norm; ten times that, for rounding, is the mark.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _case(n, loads, seed):
    from tdbem import cases
    rng = np.random.default_rng(seed)
    c = cases.make_case("cube", 1, n, [cases.Material(20.0, 0.25, 20.0)], 0.6, 1,
                        [(1.0, (1.0, 0.0, 0.0), cases.heaviside(1))] * loads, error=TOL)
    c.known[:, 1] = rng.normal(size=c.known[:, 1].shape)
    return c


def _blocks(c, sigma, seed):
    rng = np.random.default_rng(seed)
    p = c.mesh.points[c.mesh.elements[:, :4]].mean(axis=1)
    near = np.linalg.norm(p[:, None] - p[None], axis=2) < 1.6 / round((c.n_elements / 6) ** 0.5)
    i, j = np.nonzero(near)
    v = sigma * rng.normal(size=(len(i), 3, 3))
    v[i == j] += 2.0 * np.eye(3)
    E = c.n_elements
    dense = np.zeros((E, 3, E, 3))
    dense[i, :, j] = v
    rp = np.searchsorted(i, np.arange(E + 1)).astype(np.int32)
    return (rp, j.astype(np.int32), v.reshape(-1, 9)), dense.reshape(3 * E, 3 * E)


@pytest.mark.parametrize("n,loads,groups,dsm,max_leaf,sigma,precision", [
    (1, 1, 1, True, 10, 0.05, "fp64"),       # one leaf: a single CTA
    (2, 2, 1, True, 10, 0.05, "mixed"),
    (4, 1, 1, True, 1, 0.25, "fp64"),        # more columns than shared memory holds
    (4, 1, 1, False, 1, 0.25, "fp64"),
    (5, 1, 1, True, 10, 0.1, "mixed"),
    (5, 4, 4, True, 10, 0.1, "fp64"),
    (5, 4, 1, True, 3, 0.2, "fp64"),
    (5, 8, 1, True, 1, 0.25, "fp64"),
    (5, 8, 1, False, 4, 0.1, "mixed"),
    (5, 8, 1, True, 4, 0.1, "mixed"),
    (4, 16, 1, True, 10, 0.1, "fp64"),
    (4, 16, 2, True, 10, 0.1, "mixed"),
    (4, 32, 1, True, 2, 0.15, "fp64"),
    (3, 32, 1, False, 10, 0.1, "mixed"),
    (11, 1, 1, True, 7, 0.1, "fp64"),        # 726 elements: uneven ranges, halos between CTAs
])
def test_one_step_against_dense_solve(n, loads, groups, dsm, max_leaf, sigma, precision):
    from tdbem.api import MultiDomainSolver
    c = _case(n, loads, 3)
    A, Ad = _blocks(c, sigma, 4)
    K, Kd = _blocks(c, 0.1, 5)
    env = {"TDBEM_GMRES_GROUPS": str(groups), "TDBEM_GMRES_DSM": "1" if dsm else "0"}
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        s = MultiDomainSolver(c, precision=precision, n_loads=loads, max_leaf=max_leaf)
        s.load_matrices(A, K, [], [])
        lu, lt, rep = s.march(c.known)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None) if v is None else os.environ.update({k: v})
    assert rep.failed_step == 0 and rep.gmres_groups == groups
    frames = s.geometry()["transmat"].reshape(-1, 3, 3)
    s.close()
    fixed = c.bcid == 123
    mark = 10.0 * TOL * np.linalg.cond(Ad)
    for r in range(loads):
        x = np.linalg.solve(Ad, Kd @ c.known[r, 1].ravel())
        out = np.where(fixed[:, None], lt[r, 1], lu[r, 1])
        got = np.einsum("eij,ej->ei", frames, out).ravel()
        assert np.linalg.norm(got - x) <= mark * np.linalg.norm(x), (r, rep.total_inner)
    if max_leaf == 1:
        assert rep.total_inner > 32 * loads
