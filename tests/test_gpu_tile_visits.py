"""The mixed solve's tile smoother (k_tile.cu) against one launch per sweep.

Whole visits of a level on register patches, in one cluster or over the whole
grid, do the per-sweep kernels' arithmetic point by point, so a few W-cycles (the
solves are cut off after four) leave the same streamfunction bit for bit.  The
cases put
the levels' sizes on the edges of tiles and patches (odd and even columns, rows
of every remainder modulo 4, levels smaller than one tile, one tile, many), the
sweep count on the edges of the exchange period, both wall conditions, and the
per-point Chebyshev factor on a level that takes it (two levels).
"""
import os

import numpy as np
import pytest

from tracer_code_gb300 import Simulation, TracerError
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu


def _solve(p, st, fused):
    if not fused:
        os.environ["TC_NO_FUSED_VISITS"] = "1"
    try:
        g = Simulation(p)
    finally:
        os.environ.pop("TC_NO_FUSED_VISITS", None)
    with g:
        g.upload(st)
        try:
            q = g.multigrid()
        except TracerError as e:  # the cap on W-cycles; nothing else
            assert e.status == 3
            q = None
        return q, g.get("error", 1)


@pytest.mark.parametrize("nx,nz,grids,sweeps,vbc", [
    (64, 64, 4, 70, 0),     # 64, 32 and 16 columns: even, one tile and several
    (72, 40, 4, 70, 1),     # 9 x 5 coarsest; 18 x 10: odd row remainders, rigid walls
    (88, 104, 3, 69, 0),    # 22 x 26 levels, a sweep count that ends inside a period
    (100, 76, 3, 7, 1),     # 25 x 19: odd columns, few sweeps
    (200, 96, 4, 4, 0),     # one period and a remainder of one sweep
    (48, 36, 2, 70, 0),     # two levels: level 1 takes the per-point factor
    (496, 128, 5, 70, 0),   # level 1 over the whole grid
    (992, 160, 5, 11, 1),   # levels 1 and 2 over the whole grid
])
def test_tile_visits_equal_single_sweeps(gpu_lib, nx, nz, grids, sweeps, vbc):
    p = case_1024_like(nx=nx, nz=nz, grids=grids, tpc=2, Ra=1.0e4, visT=10.0)
    p.mg_zero_coarse, p.solver_precision, p.cycle_correction = 1, 1, 3
    p.aspect = nx / nz
    p.Nmulti, p.Vbc, p.max_cycles = sweeps, vbc, 4
    st = fresh_state(p, seed=nx)
    q, sf = _solve(p, st, True)
    q1, sf1 = _solve(p, st, False)
    assert q == q1
    assert np.any(sf) and np.array_equal(sf, sf1)
