"""Sweeps of deep grids, whose last blocks wait long for their first faces: results bit for bit those
of the other schedules on both sides of the depth and the width at which the sweeps keep their
instructions warm meanwhile, in 3-D and in 2-D; and on a deep, narrow grid the line sweeps of both types are
the faster ones (two to three times), so that the automatic choice takes them."""
import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu


def solver(a, grid):
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_GRID, grid)
    ilu.set_matrix(a)
    assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
    return ilu


@pytest.mark.parametrize("shape", [(10, 10, 270), (10, 10, 271), (9, 32, 249), (9, 33, 248), (5, 270, 12), (24, 24, 500),
                                   (40, 700), (40, 701)],
                         ids=lambda s: "x".join(map(str, s)))
def test_deep_grids_change_nothing(shape):
    a = g.convdiff3d(*shape) if len(shape) == 3 else g.laplace2d(*shape)
    a = g.Csr(a.n, a.row_ptr, a.col_idx, a.values * np.random.default_rng(1).uniform(0.9, 1.1, a.values.size))
    _, b = g.random_rhs(a, seed=2)
    out = {}
    for grid in (1, -1):
        ilu = solver(a, grid)
        assert ilu.info().grid_fp32 == ilu.info().grid_fp64 == (3 if grid == 1 else 0)
        x = [ilu.substitute(b) for _ in range(3)]
        assert np.array_equal(x[0], x[1]) and np.array_equal(x[0], x[2])
        gm = api.Gmres(1e-30, 20, 20)  # 20 FP32 iterations
        gm.set_preconditioner(ilu)
        gm.set_option(api.GMRES_OPT_MODE, 1)
        out[grid] = (x[0], gm.solve(a, b).x)
    assert np.array_equal(out[1][0], out[-1][0]) and np.array_equal(out[1][1], out[-1][1])


def test_deep_narrow_grids_take_the_line_sweeps():
    info = solver(g.convdiff3d(24, 24, 600), 0).info()
    assert info.grid_fp64 == 3 and info.grid_fp32 == 3
