"""LLJBASH_IluInfo describes the line-pipeline sweeps of both types, whose CTA shapes differ, and
recording their timelines changes neither."""
import numpy as np
import pytest

import bench
from par_ilu0_cpp_gb300 import api
from par_ilu0_cpp_gb300 import generators as g
from par_ilu0_cpp_gb300 import sweep_timeline

pytestmark = pytest.mark.gpu


def solver(f, **options):
    ilu = api.IluSolver()
    ilu.set_option(api.ILU_OPT_GRID, 1)
    for k, v in options.items():
        ilu.set_option(getattr(api, k), v)
    ilu.set_matrix(f)
    assert ilu.setup() == 0 and ilu.factorize() == 0, api.last_error()
    return ilu


@pytest.mark.parametrize("make", [lambda: g.convdiff3d(40, 24, 70), lambda: g.laplace2d(90, 300)], ids=["3d", "2d"])
def test_timelines_record_the_shapes_that_run(make):
    f = make()
    plain, ilu = solver(f).info(), solver(f, ILU_OPT_SWEEP_TIMELINE=1)
    gm = api.Gmres(1e-30, 5, 5)
    gm.set_preconditioner(ilu)
    gm.set_option(api.GMRES_OPT_MODE, 1)
    _, b = g.random_rhs(f, seed=1)
    gm.solve(f, b)
    ilu.substitute(b)
    for fp32 in (False, True):
        shape, used = (sweep_timeline.geometry(i, fp32) for i in (plain, ilu.info()))
        assert shape == used
        for upper in (False, True):
            tl = ilu.sweep_timeline(upper, fp32).astype(np.int64)
            assert tl.shape == (used.grid_blocks, api.LINE_TIMELINE_WORDS)
            nw = used.grid_cta_y * used.grid_cta_z
            assert (tl[:, 2:3 + nw] >= tl[:, :1]).all() and (tl[:, 0] > 0).all() and (tl[:, 3 + nw:] == 0).all()
            s = sweep_timeline.summarize(tl.astype(np.uint64), used)
            assert s["blocks"] == used.grid_blocks and s["span_us"] > 0


def test_traffic_is_looked_up_by_the_fp32_shape():
    """The benchmark's workload: the capture of the kernel that runs there is found."""
    info = solver(g.convdiff3d(128)).info()
    shape = [int(info.grid32_cta_y), int(info.grid32_cta_z), int(info.grid32_cluster)]
    for kernel in ("sptrsv_lower", "sptrsv_upper"):
        assert bench.measured_traffic(kernel, 128, 0, shape, True) is not None
