"""Warp-per-row factorisation with pivots eliminated as they become ready and quotients by
two-part reciprocals: the lane-per-row kernel's factors (which divides) bit for bit, where the
reciprocals do not apply included, and the oracle's for rows of every staging class."""
import numpy as np
import pytest

import oracle
from conftest import banded, ragged, rel_err
from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def port():
    oracle.build_port()
    return oracle.Port()


def factor(a, kernel):
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_FACTOR_KERNEL, kernel)
    ilu.set_matrix(a)
    assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
    assert ilu.info().factor_lane == (1 if kernel == 2 else 0)
    return ilu.values(), ilu.info().breakdowns, ilu.info().first_breakdown


@pytest.mark.parametrize("exponents", [0, 200, 450])
@pytest.mark.parametrize("make", [lambda: ragged(3000, 6, seed=4), lambda: banded(2000, 5, 7), lambda: g.laplace2d(50)],
                         ids=["ragged", "banded", "laplace2d"])
def test_quotients_equal_divisions(make, exponents):
    """Pivots beyond 2^+-400 and quotients beyond 2^+-600, infinities and NaNs included; entries
    of few bits, whose pivots often lie an ulp below a power of two (the Laplacian)."""
    a = make()
    rng = np.random.default_rng(exponents)
    a = g.Csr(a.n, a.row_ptr, a.col_idx, np.ldexp(a.values, rng.integers(-exponents, exponents + 1, a.values.size)))
    w, bad_w, first_w = factor(a, 2)
    for kernel in (1, 0):  # (0: the line kernel on the Laplacian)
        v, bad, first = factor(a, kernel)
        nan = np.isnan(v)
        assert np.array_equal(nan, np.isnan(w)) and np.array_equal(v[~nan].view(np.int64), w[~nan].view(np.int64))
        assert (bad, first) == (bad_w, first_w)


@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("width", [1, 15, 16, 31, 33, 70, 130])
def test_rows_of_every_length_match_the_oracle(port, width, order):
    """Rows below and above a warp's lanes, its register window and the search table's
    threshold; ready pivots in batches of 32.  A row takes up to 130 updates, each rounded
    once, of a diagonally dominant matrix: 1e-12 relative."""
    a = banded(400, width, width)
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_FACTOR_KERNEL, 1)
    ilu.set_option(api.ILU_OPT_TICKET_ORDER, order)
    ilu.set_matrix(a)
    assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
    lu_ref, _ = port.factorize(a)
    assert rel_err(ilu.values(), lu_ref, floor=1e-300) <= 1e-12
