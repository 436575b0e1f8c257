"""The viscosity filter's one-launch form (k_vis_filter) against the host loops.

Grids at both sides of its limits (17,000 points where it only smooths, 12,000 with the
eigenvalue ratio in each pass, 4,500 on stretched grids), spacings that are no powers of
two, and levels of less than a warp: every level's viscosity and,
on uniform grids, its derivatives' product in a solve (the W-cycles and SF) and the filter
counts equal those of a handle that runs the loops on the host, bit for bit.
"""
import os

import numpy as np
import pytest

from tracer_code_gb300 import Simulation, state
from tests.cases import case_1024_like, fresh_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,grids,grid", [(256, 64, 4, 0), (272, 64, 3, 0), (184, 64, 3, 0), (180, 44, 3, 0),
                                              (64, 64, 5, 0), (96, 48, 3, 1), (136, 64, 3, 1)])
def test_filter_equals_host_loops(gpu_lib, nx, nz, grids, grid):
    p = case_1024_like(nx=nx, nz=nz, tpc=3, grids=grids)
    p.aspect, p.max_cycles = nx / nz, 200
    if grid:
        p.comp, p.tracer, p.ivis = 0, 0, 2
        p.gridX, p.gridZ, p.spaceX, p.spaceZ, p.thickness, p.nbound = 1, 2, 2.0, 1.0, 0.1, 4
        st = state.initial_state(p, seed=1)
    else:
        st = fresh_state(p, seed=nx)
    out = []
    for host in (False, True):
        if host:
            os.environ["TC_HOST_LOOP"] = "1"
        try:
            g = Simulation(p)
        finally:
            os.environ.pop("TC_HOST_LOOP", None)
        g.upload(st)
        levels = range(1, g.info.grids + 1)
        for l in levels:
            g.compute_viscosity(l)
        vis = [g.get("vis_grid", l) for l in levels]
        solve = ()
        if not grid:
            q = g.multigrid()
            row = g.stats()
            solve = (q, row["n_eta"], row["eig_fine"])
        out.append((solve, vis + [g.get("vis_grid", l) for l in levels] + [g.download()["SF"]]))
        g.close()
    assert out[0][0] == out[1][0]
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)
