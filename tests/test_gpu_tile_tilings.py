"""Visits over the whole grid (k_tile.cu) of a level whose two smoothing factors take
different tilings: the uniform factor's 77 tiles and the per-point factor's 90 on 488x224
points of a GPU with 152 SMs.

The tiles number their exchanges from visit to visit, and a visit on either tiling must
find its neighbours at the same number.  Three levels: the level above the coarsest is
smoothed in both directions, with the per-point factor downwards.  Two levels: autotuning
takes the uniform factor, the solves the per-point one.  Either way a few W-cycles leave
what one launch per sweep leaves, bit for bit, in the first solve and in a later one.
"""
import os

import numpy as np
import pytest

from tracer_code_gb300 import Simulation, TracerError
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu


def _solves(p, st, fused, tune):
    if not fused:
        os.environ["TC_NO_FUSED_VISITS"] = "1"
    try:
        g = Simulation(p)
    finally:
        os.environ.pop("TC_NO_FUSED_VISITS", None)
    out = []
    with g:
        g.upload(st)
        for n in range(3):
            if tune and n < 2:  # before the first and the second solve
                tuned = g.autotune()
                # the shape the solve is to run: over the grid
                g.set_launch_shapes([(bx, by, 1) for bx, by, _ in tuned])
            try:
                q = g.multigrid()
            except TracerError as e:  # the cap on W-cycles; nothing else
                assert e.status == 3
                q = None
            out.append((q, g.get("error", 1)))
    return out


@pytest.mark.parametrize("nx,nz,grids,sweeps,tune", [(976, 448, 3, 70, False), (976, 448, 3, 11, False),
                                                     (488, 224, 2, 70, True)])
def test_visits_on_two_tilings_equal_single_sweeps(gpu_lib, nx, nz, grids, sweeps, tune):
    p = case_1024_like(nx=nx, nz=nz, grids=grids, tpc=1, Ra=1.0e4, visT=10.0)
    p.mg_zero_coarse, p.solver_precision, p.cycle_correction = 1, 1, 3
    p.aspect = nx / nz
    p.Nmulti, p.max_cycles = sweeps, 3
    st = fresh_state(p, seed=nx)
    a, b = _solves(p, st, True, tune), _solves(p, st, False, False)
    for (q, sf), (q1, sf1) in zip(a, b):
        assert q == q1
        assert np.any(sf) and np.array_equal(sf, sf1)
