"""Waits of the line kernels that run out (a limit of 1 us cuts short the waits of deep grids): the
call reports it, and with the default limit back the same solver gives the factors and the
solutions of one that never gave up, bit for bit: tickets, exchange buffers (the allocation-free
substitution has its own) and barriers are as they were."""
import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g
from test_zz_no_alloc import _DeviceArray, _cudart

pytestmark = pytest.mark.gpu

GRIDS = {"2d": (lambda: g.laplace2d(16, 9000), {}), "3d": (lambda: g.convdiff3d(6, 12, 3000), {}),
         "2d_plain": (lambda: g.laplace2d(16, 9000), {api.ILU_OPT_GRID_CLUSTER: 0}),
         "3d_plain": (lambda: g.convdiff3d(6, 12, 3000), {api.ILU_OPT_GRID_CLUSTER: 0})}


def solver(a, options):
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_GRID, 1)
    for k, v in options.items():
        ilu.set_option(k, v)
    ilu.set_matrix(a)
    assert ilu.setup() == 0, api.last_error()
    return ilu


@pytest.mark.parametrize("name", list(GRIDS))
def test_line_kernels_give_up_and_recover(name):
    make, options = GRIDS[name]
    a = make()
    _, b = g.random_rhs(a, seed=5)
    rt = _cudart()
    db, dx = _DeviceArray(rt, a.n), _DeviceArray(rt, a.n)
    db.put(b)

    def limit(us):
        ilu.set_option(api.ILU_OPT_WAIT_LIMIT_US, us)

    def no_alloc():
        if ilu.lib.LLJBASH_IluSolverSubstituteDeviceNoAlloc(ilu.h, db.ptr, dx.ptr) != 0:
            raise RuntimeError(api.last_error())
        return dx.get()

    def mixed():
        gm = api.Gmres(1e-30, 10, 10)
        gm.set_preconditioner(ilu)
        gm.set_option(api.GMRES_OPT_MODE, 1)
        res = gm.solve(a, b)
        if res.iterations == 0:  # (a solve that threw)
            raise RuntimeError(api.last_error())
        return res.x

    ilu = solver(a, options)
    assert ilu.info().grid_fp64 == 3 and ilu.info().grid_fp32 == 3
    assert ilu.factorize() == 0, api.last_error()
    lu, calls = ilu.values(), (lambda: ilu.substitute(b), no_alloc, mixed)
    want = [f() for f in calls]

    ilu = solver(a, options)
    limit(1)
    assert ilu.factorize() == -1 and "timed out" in api.last_error()
    limit(0)
    ilu.set_values(a.values)
    assert ilu.factorize() == 0, api.last_error()
    assert np.array_equal(ilu.values(), lu)
    for f, x in zip(calls, want):
        limit(1)
        try:
            out = f()
            assert name.startswith("3d") and np.array_equal(out, x)  # (3-D sweeps limit how deep a block waits)
        except RuntimeError as e:
            assert "timed out" in str(e)
        limit(0)
        for h, y in zip(calls, want):
            assert np.array_equal(h(), y)
    limit(1)
    ilu.set_values(a.values)
    assert ilu.factorize() == -1
    limit(0)
    ilu.set_values(a.values)
    assert ilu.factorize() == 0 and np.array_equal(ilu.values(), lu)
    for f, x in zip(calls, want):
        assert np.array_equal(f(), x)
    db.free()
    dx.free()
