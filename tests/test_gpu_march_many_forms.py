"""Grouped march_many where one model's vectors fit the shared memory of its GMRES
cluster and another's do not (B200): each model keeps its own form of the solver.
A model of one leaf holds the clusters to one CTA; a rod of 120 elements fits, one
of 750 with eight load cases does not (480 bytes a row and CTA in mixed precision,
of 224 KB).

In mixed precision the forms round differently (FP32 or FP64 source of the Arnoldi
product), so the small rod's results tell its form: bit for bit the same whether
the third model fits or not.  The large one's are held to its own march, 1e-7 as
in test_gpu_march_many.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOADS, NSTEP = 8, 17


def _rod(n, seed):
    from tdbem import cases
    c = cases.config_uneven_rods(count=1, nstep=NSTEP, n_min=n, n_max=n, seed=seed, error=1e-12)[0]
    rng = np.random.default_rng(11)
    c.known = np.concatenate([c.known * rng.uniform(0.5, 2.0) for _ in range(LOADS)])
    return c


def _grouped(rods, monkeypatch):
    import torch
    from tdbem.api import MultiDomainSolver, march_many
    monkeypatch.setenv("TDBEM_MARCH_MANY", "grouped")
    solvers = []
    for i, c in enumerate(rods):
        solvers.append(MultiDomainSolver(c, precision="mixed", n_loads=LOADS, max_leaf=64 if i == 0 else None))
        solvers[-1].assemble()
    known = [torch.from_numpy(np.ascontiguousarray(c.known)).cuda() for c in rods]
    lu, lt = ([torch.zeros_like(k) for k in known] for _ in range(2))
    reps = march_many(solvers, *([x.data_ptr() for x in v] for v in (known, lu, lt)),
                      torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert all(r.steps_solved == NSTEP and r.gmres_cluster == 1 for r in reps)
    return solvers, [(a.cpu().numpy(), b.cpu().numpy()) for a, b in zip(lu, lt)]


def test_models_keep_their_forms(monkeypatch):
    one, small, other, large = _rod(1, 3), _rod(2, 4), _rod(2, 5), _rod(5, 6)
    _, fit = _grouped([one, small, other], monkeypatch)
    solvers, mix = _grouped([one, small, large], monkeypatch)
    for i in range(2):
        assert np.array_equal(fit[i][0], mix[i][0]) and np.array_equal(fit[i][1], mix[i][1]), i
    u, t, _ = solvers[2].march(large.known)
    for a, b in zip(mix[2], (u, t)):
        assert np.max(np.abs(a - b)) <= 1e-7 * np.max(np.abs(b))
