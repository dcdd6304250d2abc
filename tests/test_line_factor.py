"""Line-pipeline factorisation of 7- / 5-point stencils in natural order: the factors, the
breakdown report and the shifted factors of the warp-per-row kernel bit for bit (both round
each quotient and each update once, in the same order), at partly filled lanes, warps, blocks
and clusters, and where the two-part reciprocal does not apply."""
import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu

SHAPES = [(3, 22), (64, 65), (301, 77), (1500, 33), (7, 2),  # 5-point: nx, ny
          (3, 3, 8), (3, 40, 70), (33, 5, 4), (50, 9, 65), (41, 70, 29), (300, 17, 9), (20, 100, 100)]


def stencil(shape, seed, exponents=0):
    a = g.convdiff3d(*shape) if len(shape) == 3 else g.laplace2d(*shape)
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(a.n), np.diff(a.row_ptr))
    v = rng.uniform(-1, 1, a.row_ptr[-1])
    v[rows == a.col_idx] = rng.uniform(2, 6, a.n) * rng.choice([-1, 1], a.n)
    if exponents:
        v = np.ldexp(v, rng.integers(-exponents, exponents + 1, v.size))
    return g.Csr(a.n, a.row_ptr, a.col_idx, v)


def factor(a, kernel, shift=None):
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_FACTOR_KERNEL, kernel)
    ilu.set_matrix(a)
    assert ilu.setup() == 0, api.last_error()
    out = []
    for _ in range(2):  # the second with the exchange buffers as the first left them
        ilu.set_values(a.values)
        if shift is not None:
            ilu.set_shift(shift)
        assert ilu.factorize() == 0, api.last_error()
        info = ilu.info()
        out.append((ilu.values(), info.breakdowns, info.first_breakdown))
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True) and out[0][1:] == out[1][1:]
    return out[0]


def same(x, y):
    nan = np.isnan(x)
    return np.array_equal(nan, np.isnan(y)) and np.array_equal(x[~nan].view(np.int64), y[~nan].view(np.int64))


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_factors_equal_the_row_elimination(shape):
    a = stencil(shape, seed=sum(shape))
    v, bad, first = factor(a, 0)
    w, bad_w, first_w = factor(a, 1)
    assert same(v, w) and (bad, first) == (bad_w, first_w)
    shift = np.random.default_rng(1).uniform(0.0, 0.5, a.n)
    assert same(factor(a, 0, shift)[0], factor(a, 1, shift)[0])


@pytest.mark.parametrize("exponents", [200, 450])
@pytest.mark.parametrize("shape", [(40, 33), (20, 11, 13)], ids=lambda s: "x".join(map(str, s)))
def test_pivots_and_quotients_out_of_range(shape, exponents):
    """Pivots beyond 2^+-400 and quotients beyond 2^+-600, infinities and NaNs included."""
    a = stencil(shape, seed=5, exponents=exponents)
    v, bad, first = factor(a, 0)
    w, bad_w, first_w = factor(a, 1)
    assert same(v, w) and (bad, first) == (bad_w, first_w)


@pytest.mark.parametrize("shape,row", [((64, 40), 0), ((64, 40), 1000), ((12, 20, 30), 4321)])
def test_zero_pivot_is_reported(shape, row):
    """A zero diagonal in a row without lower couplings is a zero pivot."""
    a = stencil(shape, seed=3)
    v = a.values.copy()
    lo, hi = a.row_ptr[row], a.row_ptr[row + 1]
    v[lo:hi][a.col_idx[lo:hi] <= row] = 0.0
    a = g.Csr(a.n, a.row_ptr, a.col_idx, v)
    v, bad, first = factor(a, 0)
    w, bad_w, first_w = factor(a, 1)
    assert first == row and (bad, first) == (bad_w, first_w) and same(v, w)


def test_more_blocks_than_resident_ctas():
    a = stencil((12, 420, 400), seed=8)
    v = factor(a, 0)[0]
    assert same(v, factor(a, 1)[0])


def test_packs_follow_the_chosen_sweeps():
    """After the sweeps are chosen, later factorisations fill only the packs that they read:
    substitution and its allocation-free form see the new factors."""
    a = stencil((30, 31, 32), seed=9)
    b = np.random.default_rng(2).uniform(-1, 1, a.n)
    ref = api.IluSolver()
    ref.set_option(api.ILU_OPT_GRID, -1)
    ref.set_matrix(a)
    assert ref.setup() == 0 and ref.factorize() == 0
    ilu = api.IluSolver()
    ilu.set_matrix(a)
    assert ilu.setup() == 0
    for seed in (9, 10, 11):
        new = stencil((30, 31, 32), seed=seed)
        for s in (ref, ilu):
            s.set_values(new.values)
            assert s.factorize() == 0, api.last_error()
        assert np.array_equal(ref.substitute(b), ilu.substitute(b))
