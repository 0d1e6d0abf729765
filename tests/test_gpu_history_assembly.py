"""History and step-0 matrices assembled over all steps of a pair at once, against
the C oracle's step-by-step assembly (B200): domains of one element a face, of 96
elements (more sources than a CTA's 64, not a multiple), several materials, and
time steps short and long against the element size (waves that stay many steps in
an element, or cross it within one), with the workspace limit cutting the rows
into ranges; and the material gradient's walk over the same steps.

Matrices: 1e-12 relative to the largest entry, as elsewhere; a block is stored
when an entry exceeds 1e-14, so one that only one side stores may reach 2e-14.
Gradient: scaling all E and rho by one factor changes no wave speed, so
sum_d (E_d dJ/dE_d + rho_d dJ/drho_d) = -<dJ/dU, U> exactly; held to 1e-9, where
GMRES stops at 1e-14.
"""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(3, 1, 0.6), (3, 1, 0.1), (2, 3, 2.5), (2, 4, 0.6), (1, 5, 0.9)]


def _case(domains, n, beta, nstep):
    from tdbem import cases
    rng = np.random.default_rng(100 * domains + n)
    mats = [cases.Material(rng.uniform(15, 30), rng.uniform(0.15, 0.35), rng.uniform(15, 25)) for _ in range(domains)]
    return cases.make_case("pairs", domains, n, mats, beta, nstep, [(1.0, (0.3, 0.9, 0.4), cases.heaviside(nstep))],
                           error=1e-14)


def _blocks(m):
    rp, col, val = m
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    return {(int(r), int(c)): v for r, c, v in zip(rows, col, np.asarray(val).reshape(-1, 9))}


@pytest.mark.parametrize("domains,n,beta", SHAPES)
def test_history_matrices_equal_the_oracle(domains, n, beta):
    from tdbem.api import MultiDomainSolver
    from oracle_lib import Oracle
    c = _case(domains, n, beta, 40)
    o = Oracle(c)
    o.assemble()
    s = MultiDomainSolver(c)
    s.assemble()
    last = s.march(c.known[0])[2].history_steps
    present = [k for k in range(1, o.history_step_bound() + 1) if k <= last]
    assert present
    limits = {}
    for limit in ("1", "100000"):
        os.environ["TDBEM_HISTORY_SCRATCH"] = limit
        try:
            limits[limit] = MultiDomainSolver(c)
            limits[limit].assemble()
        finally:
            os.environ.pop("TDBEM_HISTORY_SCRATCH")
    for k in present:
        for name in ("MTS", "MGS"):
            got = s.export_matrix(name, k)
            for t in limits.values():
                for a, b in zip(t.export_matrix(name, k), got):
                    assert np.array_equal(a, b), (name, k)
            a, b = _blocks(got), _blocks(o.matrix(name, k))
            if not b:
                assert not a or max(np.max(np.abs(v)) for v in a.values()) <= 2e-14, (name, k)
                continue
            mark = max(1e-12 * max(np.max(np.abs(v)) for v in b.values()), 2e-14)
            zero = np.zeros(9)
            for key in a.keys() | b.keys():
                assert np.max(np.abs(a.get(key, zero) - b.get(key, zero))) <= mark, (name, k, key)


@pytest.mark.parametrize("domains,n,beta", SHAPES)
def test_step0_matrices_equal_the_oracle(domains, n, beta):
    from tdbem.api import MultiDomainSolver
    from oracle_lib import Oracle
    c = _case(domains, n, beta, 4)
    o = Oracle(c)
    o.assemble()
    s = MultiDomainSolver(c)
    s.assemble()
    for name in ("A", "KnownM"):
        a, b = _blocks(s.export_matrix(name)), _blocks(o.matrix(name))
        mark = max(1e-12 * max(np.max(np.abs(v)) for v in b.values()), 2e-14)
        zero = np.zeros(9)
        for key in a.keys() | b.keys():
            assert np.max(np.abs(a.get(key, zero) - b.get(key, zero))) <= mark, (name, key)


@pytest.mark.parametrize("domains,n,beta", SHAPES)
def test_material_gradient_scaling_identity(domains, n, beta):
    from tdbem.api import MultiDomainSolver
    c = _case(domains, n, beta, 24)
    s = MultiDomainSolver(c)
    s.assemble()
    lu, _, rep = s.march_forward(c.known[0])
    assert rep.failed_step == 0
    cot = np.random.default_rng(5).normal(size=lu.shape)
    cot[0] = 0.0
    _, gm, _ = s.march_backward(cot, None)
    E, rho = np.array([m.E for m in c.materials]), np.array([m.rho for m in c.materials])
    lhs, rhs = E @ gm[:, 0] + rho @ gm[:, 1], -np.sum(cot * lu)
    assert abs(lhs - rhs) <= 1e-9 * np.sum(np.abs(cot * lu)), (lhs, rhs)
