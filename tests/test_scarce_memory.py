"""Device memory that holds what a factor cannot do without but not the line kernels' operand
streams: set-up takes the other schedules and kernels instead of failing, with the same factors and
solutions.  And the line factorisation takes no memory of its own beside the line sweeps."""
import ctypes

import numpy as np
import pytest

from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g
from test_zz_no_alloc import _cudart

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes(rt):
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    assert rt.cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def run(rt, a, b, options, after_setup=None):
    """Bytes that set-up takes, info, factors and solution."""
    ilu = api.IluSolver()
    for k, v in options.items():
        ilu.set_option(k, v)
    ilu.set_matrix(a)
    before = free_bytes(rt)
    assert ilu.setup() == 0, api.last_error()
    taken = before - free_bytes(rt)
    if after_setup is not None:
        after_setup()
    assert ilu.factorize() == 0, api.last_error()
    return taken, ilu.info(), ilu.values(), ilu.substitute(b)


def test_setup_without_room_for_the_line_kernels():
    rt = _cudart()
    a = g.convdiff3d(128, 120, 112)
    _, b = g.random_rhs(a, seed=1)
    _, info, lu, x = run(rt, a, b, {})
    assert info.grid_fp64 == 3 and info.grid_fp32 == 3
    need = run(rt, a, b, {api.ILU_OPT_GRID: -1})[0]
    hog = ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(hog), free_bytes(rt) - need - 56 * MB) == 0
    released = []

    def release():
        rt.cudaFree(hog)
        released.append(True)

    try:
        _, info, lu2, x2 = run(rt, a, b, {}, after_setup=release)
    finally:
        if not released:
            release()
    assert info.grid_fp64 == 0 and info.grid_fp32 == 0
    assert np.array_equal(lu, lu2) and np.array_equal(x, x2)


def test_line_factorisation_shares_the_sweeps_streams():
    rt = _cudart()
    a = g.convdiff3d(96)
    _, b = g.random_rhs(a, seed=1)
    run(rt, a, b, {})
    line = run(rt, a, b, {})[0]
    rows = run(rt, a, b, {api.ILU_OPT_FACTOR_KERNEL: 1})[0]
    # (64 B per row would be 54 MB; the other kernel keeps 16 B per row, the line's faces are 5 MB)
    assert line <= rows + 8 * MB
