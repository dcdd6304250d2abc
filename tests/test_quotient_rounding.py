"""Quotients by two-part reciprocals (FP64 backward sweeps and factorisations) at dividends and
divisors whose quotient lies next to the middle between two numbers: correctly rounded, as the
division operator gives them, in every bit.

For an odd 53-bit divisor d and a small odd r, a 2^(s + 1) = r (mod d) makes a / d lie r / (2 d)
units in the last place from such a middle, for the a of 53 bits (s = 52: a >= d, 53: a < d).
Nearer than 1 / (2 d) no quotient comes."""
import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu

LO, HI = 1 << 52, 1 << 53
# dividend, divisor: short significands and their neighbours
PAIRS = [(5525790499943899.0, 6902488716921435.0),
         (float.fromhex("0x1.1000000000002p+0"), float.fromhex("0x1.8000000000003p+0")),
         (float.fromhex("0x1.12ffffffffffep+0"), float.fromhex("0x1.5fffffffffffdp+0")),
         (1.0, 1.0 - 2.0**-53), (1.5, 1.0 + 2.0**-52), (1.25, 1.0 - 2.0**-53), (1.0, 1.0 + 2.0**-52)]


def dividends(d, residues):
    """Dividends a (53-bit integers) of the odd divisor d with a / d next to a middle."""
    out = []
    for s in (52, 53):
        inv = pow(pow(2, s + 1, d), -1, d)
        for r in residues:
            a = r * inv % d
            for a in (a, a + d):
                if LO <= a < HI and (a >= d) == (s == 52):
                    out.append(a)
    return out


def pool(rng, count):
    """(divisor, its dividends) for `count` divisors: random ones, and neighbours of numbers of few
    bits."""
    found = []
    while len(found) < count:
        if len(found) % 2:
            d = int(rng.integers(LO, HI)) | 1
        else:
            top = int(rng.integers(8, 17))  # 4 bits
            d = (top << 49) + int(rng.integers(-64, 64)) | 1
            if not LO <= d < HI:
                continue
        residues = [int(r) * int(s) for r in (1, 3, 5, 2 * int(rng.integers(3, 1000)) + 1) for s in (1, -1)]
        a = dividends(d, residues)
        if a:
            found.append((d, a))
    return found


def scaled(rng, v, spread):
    v = np.asarray(v, dtype=np.float64) * rng.choice([-1.0, 1.0], len(v))
    return np.ldexp(v, rng.integers(-spread, spread + 1, len(v)) - 52)


def same_bits(x, y):
    return np.array_equal(x.view(np.int64), y.view(np.int64))


SWEEPS = {
    "line": (lambda: g.laplace2d(70, 90), {api.ILU_OPT_GRID: 1}),
    "line_3d": (lambda: g.convdiff3d(20, 18, 17), {api.ILU_OPT_GRID: 1}),
    "blocks": (lambda: g.laplace2d(70, 90), {api.ILU_OPT_GRID: -1}),
    "levels": (lambda: g.laplace2d(70, 90), {api.ILU_OPT_GRID: -1, api.ILU_OPT_BLOCK_ROWS: -1}),
    "lane_groups": (lambda: g.lognormal27(18, seed=1), {api.ILU_OPT_GRID: -1, api.ILU_OPT_BLOCK_ROWS: -1,
                                                        api.ILU_OPT_ROW_LANES: 8}),
}


@pytest.mark.parametrize("name", list(SWEEPS))
def test_backward_sweep_quotients(name):
    """Diagonal values on the pattern: the backward sweep leaves b / d."""
    make, options = SWEEPS[name]
    a = make()
    rng = np.random.default_rng(len(name))
    rows = np.repeat(np.arange(a.n), np.diff(a.row_ptr))
    pairs = [(x, d) for d, xs in pool(rng, 3000) for x in xs]
    pick = rng.integers(0, len(pairs), a.n)
    b = scaled(rng, [pairs[i][0] for i in pick], 150)
    d = scaled(rng, [pairs[i][1] for i in pick], 150)
    for i, (x, y) in enumerate(PAIRS):
        b[7 * i], d[7 * i] = x, y
    values = np.where(a.col_idx == rows, d[rows], 0.0)
    ilu = api.IluSolver()
    for k, v in options.items():
        ilu.set_option(k, v)
    ilu.set_matrix(g.Csr(a.n, a.row_ptr, a.col_idx, values))
    assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
    assert ilu.info().grid_fp64 == (3 if name.startswith("line") else 0)
    assert same_bits(ilu.substitute(b), b / d)


@pytest.mark.parametrize("kernel,order", [(0, 0), (1, 0), (1, 2)], ids=["line", "rows", "subtrees"])
@pytest.mark.parametrize("make", [lambda: g.laplace2d(60, 50), lambda: g.convdiff3d(15, 13, 16)], ids=["2d", "3d"])
def test_factorisation_quotients(make, kernel, order):
    """Lower triangular values on the stencil: l_ij = a_ij / a_jj."""
    a = make()
    rng = np.random.default_rng(a.n)
    rows = np.repeat(np.arange(a.n), np.diff(a.row_ptr))
    div = pool(rng, 2000)
    pick = rng.integers(0, len(div), a.n)
    d = scaled(rng, [div[i][0] for i in pick], 150)
    values = np.zeros(a.row_ptr[-1])
    values[rows == a.col_idx] = d
    low = a.col_idx < rows
    lists = [div[pick[j]][1] for j in a.col_idx[low]]
    values[low] = scaled(rng, [x[int(rng.integers(0, len(x)))] for x in lists], 150)
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_FACTOR_KERNEL, kernel)
    ilu.set_option(api.ILU_OPT_TICKET_ORDER, order)
    ilu.set_matrix(g.Csr(a.n, a.row_ptr, a.col_idx, values))
    assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
    want = values.copy()
    want[low] = values[low] / d[a.col_idx[low]]
    assert same_bits(ilu.values(), want)
