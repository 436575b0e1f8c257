"""The give-up exits of the tile visits (k_tile.cu) over the whole grid and in one cluster.

With the debug switch of test_gpu_timeouts.py every visit gives up before its first
exchange: the solve returns TC_ERR_DEVICE_TIMEOUT.  With it off the same handle then
solves with the bits of a fresh one, twice, which needs the tiles' exchange numbers to
have stayed in step.  496x128: level 1 over the grid; 256x16 with two levels: the
per-point factor in a cluster; 992x160: two levels over the grid.  (Coarse bands of at most
kl = 20: their factorisation has no such waits.)
"""
import numpy as np
import pytest

from tracer_code_gb300 import Simulation, TracerError
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu

TIMEOUT = 13  # TC_ERR_DEVICE_TIMEOUT


@pytest.mark.parametrize("nx,nz,grids", [(496, 128, 5), (256, 16, 2), (992, 160, 5), (256, 64, 4)])
def test_visit_gives_up_then_handle_solves(gpu_lib, nx, nz, grids):
    p = case_1024_like(nx=nx, nz=nz, grids=grids, tpc=1, Ra=1.0e4, visT=10.0)
    p.mg_zero_coarse, p.solver_precision, p.cycle_correction = 1, 1, 3
    p.aspect, p.max_cycles = nx / nz, 60
    st = fresh_state(p, seed=nx)

    def solves(g):
        return [(g.multigrid(), g.get("error", 1)) for _ in range(2)]

    with Simulation(p) as f:
        f.upload(st)
        ref = solves(f)
    with Simulation(p) as g:
        g.upload(st)
        for _ in range(2):
            g.debug_wait_test(True)
            with pytest.raises(TracerError) as e:
                g.multigrid()
            assert e.value.status == TIMEOUT
        g.debug_wait_test(False)
        out = solves(g)
    for (q, sf), (q1, sf1) in zip(out, ref):
        assert q == q1
        assert np.any(sf) and np.array_equal(sf, sf1)
