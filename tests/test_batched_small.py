"""Batches on both sides of the size up to which the batched solver takes its variant for small
systems (576, 400 and 200 rows for 1, 4 and 16 right-hand sides per item): every answer meets
the FP64 residual tolerance, in batches of equal and of uneven systems."""
import numpy as np
import pytest

from conftest import ragged
from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,limit", [(1, 576), (4, 400), (16, 200)])
@pytest.mark.parametrize("over", [0, 1])
def test_answers_around_the_small_limit(lanes, limit, over):
    systems = [ragged(limit + over, 4, seed=1), g.laplace2d(9, 7), g.laplace2d(1, 1), g.convdiff3d(5, 4, 6), ragged(37, 9, seed=2)]
    systems += [g.laplace2d(4 + i % 9, 11 - i % 7) for i in range(60)]
    rng = np.random.default_rng(limit + over)
    for nrhs in (1, 5):
        bs = [rng.uniform(-1, 1, (nrhs, a.n)) for a in systems]
        solver = api.BatchSolver(systems, nrhs=nrhs, restart=30)
        solver.set_shape(2, True, lanes)
        out = solver.solve(np.concatenate([b.ravel() for b in bs]))
        assert out["converged"].all()
        pos = 0
        for a, b in zip(systems, bs):
            for r in range(nrhs):
                x = out["x"][pos:pos + a.n]
                pos += a.n
                assert np.linalg.norm(b[r] - g.spmv(a, x)) <= 1.0001e-8 * np.linalg.norm(b[r])
