"""The factorisation kernel that runs, as LLJBASH_IluInfo reports it: the line pipeline on every full
stencil of at least three cells along x (and y in 3-D) unless another kernel, ticket order or
schedule is asked for; and two lines only, the narrowest grid it takes."""
import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g
from test_line_factor import SHAPES, factor, same, stencil

pytestmark = pytest.mark.gpu


def info(a, options=()):
    ilu = api.IluSolver()
    for k, v in options:
        ilu.set_option(k, v)
    ilu.set_matrix(a)
    assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
    return ilu.info()


@pytest.mark.parametrize("shape", [s for s in SHAPES if np.prod(s) >= 64] + [(40, 2), (40, 33), (20, 11, 13), (64, 40),
                                                                              (12, 20, 30), (12, 420, 400), (30, 31, 32)],
                         ids=lambda s: "x".join(map(str, s)))
def test_full_stencils_run_on_the_line_pipeline(shape):
    i = info(stencil(shape, seed=1))
    assert (i.factor_line, i.factor_lane) == (1, 0)
    assert info(stencil(shape, seed=1), [(api.ILU_OPT_FACTOR_KERNEL, 1)]).factor_line == 0


@pytest.mark.parametrize("shape", [(7, 2), (2, 60, 60), (60, 2, 60), (2, 200)], ids=lambda s: "x".join(map(str, s)))
def test_grids_that_elimination_couples_do_not(shape):
    assert info(stencil(shape, seed=1)).factor_line == 0


@pytest.mark.parametrize("options", [[(api.ILU_OPT_FACTOR_KERNEL, 2)], [(api.ILU_OPT_TICKET_ORDER, 1)],
                                     [(api.ILU_OPT_TICKET_ORDER, 2)], [(api.ILU_OPT_GRID, -1)],
                                     [(api.ILU_OPT_BLOCK_ROWS, 512)], [(api.ILU_OPT_BLOCK_ROWS, -1)]], ids=str)
def test_requests_for_other_kernels_are_kept(options):
    assert info(stencil((20, 11, 13), seed=1), options).factor_line == 0


@pytest.mark.parametrize("nx,line", [(910, 1), (911, 0)])
def test_longest_grid_lines(nx, line):
    """The last line whose faces fit in a CTA's shared memory, and the next, which the other kernel
    takes, with the same factors."""
    a = stencil((nx, 5, 3), seed=2)
    assert info(a).factor_line == line
    assert same(factor(a, 0)[0], factor(a, 1)[0])


def test_other_patterns_do_not():
    assert info(g.lognormal27(8, seed=1)).factor_line == 0
    assert info(api.iluk_symbolic(g.laplace2d(30), 1)[0]).factor_line == 0


def test_two_lines():
    a = stencil((40, 2), seed=4)
    v, bad, first = factor(a, 0)
    w, bad_w, first_w = factor(a, 1)
    assert same(v, w) and (bad, first) == (bad_w, first_w)
