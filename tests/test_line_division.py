"""FP64 backward line sweep: the quotient by a two-part reciprocal (line_quotient) where it can
go wrong — divisors and quotients outside its range, subnormal results, exact zeros of both
signs, infinities and NaN — and the face waits of grids whose sides leave partly filled
warps, chunks of steps and blocks.  The level-ordered kernel divides with the division
operator, so both must agree in every bit (NaN in the same places)."""
import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu


def solver(f, grid, block_rows=0):
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_GRID, grid)
    ilu.set_option(api.ILU_OPT_BLOCK_ROWS, block_rows)
    ilu.set_matrix(f)
    assert ilu.setup() == 0, api.last_error()
    assert ilu.factorize() == 0, api.last_error()
    return ilu


def scaled_columns(a, rng, exponents):
    """A D with D = 10^e: the factors' L is that of A, column j of U is scaled by D_j."""
    d = 10.0 ** rng.choice(exponents, a.n)
    return g.Csr(a.n, a.row_ptr, a.col_idx, a.values * d[a.col_idx])


def same_bits(x, y):
    nan = np.isnan(y)
    return np.array_equal(np.isnan(x), nan) and np.array_equal(x[~nan].view(np.int64), y[~nan].view(np.int64))


MATRICES = [lambda: g.convdiff3d(17, 9, 6), lambda: g.convdiff3d(8, 33, 5), lambda: g.laplace2d(25, 41)]


@pytest.mark.parametrize("make", MATRICES, ids=["17x9x6", "8x33x5", "2d_25x41"])
@pytest.mark.parametrize("exponents", [(0,), (-3, 0, 2), (-119, 0, 119), (-125, 0, 125), (-140, 140)],
                         ids=["plain", "mild", "inside", "outside", "far"])
def test_quotients_match_the_division(make, exponents):
    a = make()
    rng = np.random.default_rng(len(exponents) + abs(exponents[0]))
    f = scaled_columns(a, rng, exponents)
    line, ref = solver(f, 1), solver(f, -1, -1)
    assert line.info().grid_fp64 == 3 and ref.info().grid_fp64 == 0
    dense = rng.uniform(-1, 1, a.n)
    point = np.zeros(a.n)
    point[a.n // 3] = -1.0
    zeros = np.where(rng.random(a.n) < 0.5, 0.0, -0.0)
    odd = dense.copy()
    odd[a.n // 2] = np.inf
    odd[a.n // 4] = np.nan
    for b in (dense, dense * 1e-170, dense * 1e150, dense * 5e-310, point, zeros, odd):
        x = ref.substitute(b)
        assert same_bits(line.substitute(b), x)
        assert same_bits(line.substitute(b), x)  # the exchange buffers are back at the sentinel


def test_random_quotients_match_the_division():
    """Two million quotients per call: a two-entry chain per line leaves the division of
    random dividends by random divisors."""
    nx, nz = 1000, 2000
    n = nx * nz
    rng = np.random.default_rng(3)
    a = g.laplace2d(nx, nz)
    rows = np.repeat(np.arange(n), np.diff(a.row_ptr))
    v = np.where(a.col_idx == rows, rng.uniform(1, 2, n)[rows] * 2.0 ** rng.integers(-300, 300, n)[rows], 0.0)
    f = g.Csr(n, a.row_ptr, a.col_idx, v)  # diagonal values on the stencil's pattern
    line = solver(f, 1)
    assert line.info().grid_fp64 == 3
    d = v[a.col_idx == rows]
    for _ in range(3):
        b = rng.uniform(1, 2, n) * 2.0 ** rng.integers(-300, 300, n)
        assert same_bits(line.substitute(b), b / d)
