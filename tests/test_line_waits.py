"""Sweeps whose blocks wait long for their first faces (they run their first chunk on an idle
area meanwhile): results bit for bit those of the other schedules, on both sides of the grid
size where FP32 sweeps start to do so and with partly filled last warps."""
import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(400, 300), (400, 301), (37, 1100), (701, 650)])
def test_long_waits_change_nothing(nx, nz):
    a = g.laplace2d(nx, nz)
    a = g.Csr(a.n, a.row_ptr, a.col_idx, a.values * np.random.default_rng(nx).uniform(0.9, 1.1, a.values.size))
    _, b = g.random_rhs(a, seed=nz)
    out = {}
    for grid in (1, -1):
        ilu = api.IluSolver()
        ilu.set_option(api.ILU_OPT_GRID, grid)
        ilu.set_matrix(a)
        assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
        assert ilu.info().grid_fp32 == ilu.info().grid_fp64 == (3 if grid == 1 else 0)
        x = [ilu.substitute(b) for _ in range(3)]
        assert np.array_equal(x[0], x[1]) and np.array_equal(x[0], x[2])
        gm = api.Gmres(1e-30, 20, 20)  # 20 FP32 iterations
        gm.set_preconditioner(ilu)
        gm.set_option(api.GMRES_OPT_MODE, 1)
        out[grid] = (x[0], gm.solve(a, b).x)
    assert np.array_equal(out[1][0], out[-1][0]) and np.array_equal(out[1][1], out[-1][1])
