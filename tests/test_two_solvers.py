"""Two solvers alive at the same time, the one whose kernels need less shared memory set up
last: a kernel's limit of dynamic shared memory (and its leave to run in clusters of more than
8 CTAs) belongs to the kernel, not to a solver, so the first solver still factorises,
substitutes and iterates afterwards, with the results that it had before."""
import numpy as np
import pytest

from conftest import banded
from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu

GRID = {api.ILU_OPT_GRID: 1}
NO_CLUSTER = {api.ILU_OPT_GRID: 1, api.ILU_OPT_GRID_CLUSTER: 0}


def blocks(rows):
    return {api.ILU_OPT_GRID: -1, api.ILU_OPT_BLOCK_ROWS: rows}


ROWS = {api.ILU_OPT_FACTOR_KERNEL: 1}
TREE = {api.ILU_OPT_FACTOR_KERNEL: 1, api.ILU_OPT_TICKET_ORDER: 2}
CASES = {
    "line_2d": (lambda: g.laplace2d(384, 70), GRID, lambda: g.laplace2d(63, 70), GRID),
    "line_2d_plain": (lambda: g.laplace2d(384, 70), NO_CLUSTER, lambda: g.laplace2d(63, 70), NO_CLUSTER),
    "line_3d": (lambda: g.convdiff3d(160, 20, 24), GRID, lambda: g.convdiff3d(12, 20, 24), GRID),
    "line_3d_plain": (lambda: g.convdiff3d(160, 20, 24), NO_CLUSTER, lambda: g.convdiff3d(12, 20, 24), NO_CLUSTER),
    "blocks": (lambda: g.convdiff3d(40), blocks(8192), lambda: g.convdiff3d(20), blocks(2048)),
    "blocks_in_clusters": (lambda: g.laplace2d(300), blocks(2048), lambda: g.laplace2d(90), blocks(1024)),
    "row_factor": (lambda: banded(400, 130, 1), ROWS, lambda: banded(300, 70, 2), ROWS),
    "subtree_factor": (lambda: banded(400, 130, 1), TREE, lambda: banded(300, 70, 2), TREE),
}


def solver(a, options):
    ilu = api.IluSolver()
    for k, v in options.items():
        ilu.set_option(k, v)
    ilu.set_matrix(a)
    assert ilu.setup() == 0, api.last_error()
    return ilu


def results(ilu, a, b):
    ilu.set_values(a.values)
    assert ilu.factorize() == 0, api.last_error()
    gm = api.Gmres(1e-30, 8, 8)
    gm.set_preconditioner(ilu)
    gm.set_option(api.GMRES_OPT_MODE, 1)  # FP32 sweeps
    return ilu.values(), ilu.substitute(b), gm.solve(a, b).x


@pytest.mark.parametrize("name", list(CASES))
def test_smaller_solver_set_up_last(name):
    make, options, make_small, small_options = CASES[name]
    a, s = make(), make_small()
    _, b = g.random_rhs(a, seed=3)
    _, bs = g.random_rhs(s, seed=4)
    first = solver(a, options)
    before = results(first, a, b)
    second = solver(s, small_options)
    results(second, s, bs)
    for x, y in zip(results(first, a, b), before):
        assert np.array_equal(x, y)
