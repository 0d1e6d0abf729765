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


def test_failed_load():
    """A load refused for its input leaves the handle with the matrices it had; one
    that fails later leaves it without any, until the next one succeeds."""
    from tdbem.api import MultiDomainSolver, TdbemError
    c = _case(8, NSTEP)
    good, other = _seeded(c.n_elements, 5, 1), _seeded(c.n_elements, 9, 2)
    s = MultiDomainSolver(c, n_loads=8)
    s.load_matrices(*good)
    ref = s.march(c.known)[:2]
    bad = [*other[:2], [(r, np.where(k == 8, j + c.n_elements * 2, j), v) for k, (r, j, v) in enumerate(other[2])],
           other[3]]
    with pytest.raises(TdbemError, match="MTS column out of range"):
        s.load_matrices(*bad)
    for a, b in zip(s.march(c.known)[:2], ref):
        assert np.array_equal(a, b)
    singular = [(other[0][0], other[0][1], 0.0 * other[0][2]), *other[1:]]
    with pytest.raises(TdbemError, match="SINGULAR_BLOCK"):
        s.load_matrices(*singular)
    with pytest.raises(TdbemError, match="NOT_ASSEMBLED"):
        s.march(c.known)
    s.load_matrices(*good)
    for a, b in zip(s.march(c.known)[:2], ref):
        assert np.array_equal(a, b)
    s.close()
