"""Batched solver on systems that leave the usual path of a level: rows of more entries than
are read ahead (27-point, ragged), levels of more rows than the CTA takes at once (a diagonal
matrix, a wide 3-D grid with 16 right-hand sides), fewer levels than the pipeline is deep."""
import numpy as np
import pytest

from conftest import ragged
from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu


def diagonal(n):
    return g.Csr(n, np.arange(n + 1), np.arange(n), np.linspace(1.0, 2.0, n))


@pytest.mark.parametrize("nrhs", [1, 4, 16])
@pytest.mark.parametrize("make", [
    lambda: [g.lognormal27(7, 6, 5), g.laplace2d(9, 4)],
    lambda: [ragged(700, 7, seed=2), g.laplace2d(2, 2)],
    lambda: [diagonal(2000), diagonal(1), g.laplace2d(40, 3)],
    lambda: [g.convdiff3d(24, 20, 18)],
], ids=["27point", "ragged", "few_levels", "wide"])
def test_every_answer_meets_the_residual(make, nrhs):
    systems = make()
    rng = np.random.default_rng(nrhs)
    bs = [rng.uniform(-1, 1, (nrhs, a.n)) for a in systems]
    out = api.BatchSolver(systems, nrhs=nrhs, restart=30).solve(np.concatenate([b.ravel() for b in bs]))
    assert out["converged"].all()
    pos = 0
    for a, b in zip(systems, bs):
        for r in range(nrhs):
            x = out["x"][pos:pos + a.n]
            pos += a.n
            assert np.linalg.norm(b[r] - g.spmv(a, x)) <= 1.0001e-8 * np.linalg.norm(b[r])
