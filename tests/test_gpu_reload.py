"""A handle that takes its matrices anew (B200): nothing of the old ones is left in
the march, the adjoint or the solver, and a load that fails leaves no handle that
marches with half of them.
"""
import numpy as np
import pytest

from test_gpu_nonfinite import _case, _matrices

pytestmark = pytest.mark.gpu

NSTEP = 12


def _seeded(E, K, seed):
    m = _matrices(E, K, 0.3)
    rng = np.random.default_rng(seed)
    scale = lambda a: (a[0], a[1], a[2] * rng.uniform(0.8, 1.2))
    return [scale(m[0]), scale(m[1]), [scale(x) for x in m[2]], [scale(x) for x in m[3]]]


def test_adjoint_follows_the_matrices():
    from tdbem.api import MultiDomainSolver
    c = _case(1, NSTEP)
    rng = np.random.default_rng(2)
    cot = rng.normal(size=(NSTEP + 1, c.n_elements, 3))
    first, second = _seeded(c.n_elements, 5, 1), _seeded(c.n_elements, 5, 2)
    out = []
    for loads in ((first, second), (second,)):
        s = MultiDomainSolver(c)
        for m in loads:
            s.load_matrices(*m)
            lu, lt, _ = s.march(c.known[0])
            g, _ = s.march_vjp(cot, -0.5 * cot)
        s.close()
        out.append((lu, lt, g))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
